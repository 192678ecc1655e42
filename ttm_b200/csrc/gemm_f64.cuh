// FP64 slice-GEMM on the double-precision matrix instruction (mma.sync m8n8k4.f64).
//
// One tile is BM (128 or 64) rows (flattened (k, i) pairs) x up to 8 * NF columns j; 2 BM threads.
// Warp w owns rows [16 w, 16 w + 16) and every column of the tile: the widths are whole builds in
// groups of eight columns, so that no warp multiplies padding (m = 100: two tiles of 56 columns).
// A and B tiles of 16 l go through a ring of ST shared-memory stages filled with cp.async.
//
// What bounds it: the FP64 pipe (37.1 TFLOP/s for a stream of mma on this part, 33.9 for plain
// DFMA) once m passes about 24; below that, reading A. A k-step of four l costs a warp 1 or 2 A and
// NF B shared loads for 2 NF mma of 256 multiply-adds each; the DFMA tile of 64 x 64 it replaced
// needed 8 loads for 16 DFMA of 32. Measured, before -> now: A 256^3, m = 128, middle mode
// 323 -> 139 us (31 TFLOP/s); (150, 171, 333), m = 100 189 -> 82 us; (200, 180, 160), m = 20
// 84 -> 19 us; contiguous fibres of 384, 78000 rows, m = 16 (TMA row kernel) 139 -> 50 us. (Running
// pointers in place of addresses recomputed per copy gave 5-15 % of that.)
// Rows of 64 for at most 16 columns with 16-byte copies (five blocks of 128 threads per SM, four for
// contiguous fibres): 59 us at 128 rows against 53; with 8-byte copies 128 rows are faster (73 against
// 119 us).
#pragma once

#include "common.cuh"

namespace tlibttm {
namespace f64 {

constexpr int BK = 16;

// Row pitches are 4 mod 16 doubles: the 4 l x 4 rows (or columns) that half a warp reads lie in
// distinct banks.
template <int BM, int NF, int ST, bool AK, bool BCM>
struct Smem {
    static constexpr int BN = NF * 8;
    static constexpr int AP = AK ? BK + 4 : BM + 4, AR = AK ? BM : BK;
    static constexpr int BP = BCM ? BN + 4 : BK + 4, BR = BCM ? BK : BN;
    __align__(16) double a[ST][AR][AP];   // [row][l] for contiguous fibres, else [l][row]
    __align__(16) double b[ST][BR][BP];   // [l][j] for column-major B, else [j][l]
};

__device__ __forceinline__ void mma(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// The first of a chain: c = a b.
__device__ __forceinline__ void mma_open(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
                 : "=d"(c[0]), "=d"(c[1])
                 : "d"(a), "d"(b), "d"(0.0));
}

// Copies 16 or 8 bytes; zeroes the destination where !ok (src is then not read).
__device__ __forceinline__ void copy16(void* dst, const void* src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 8 : 0)
                 : "memory");
}

// Builds for m <= 16 that take problems from kernels with several short chains (FOLD, the chains' length;
// 0: one chain) add up in levels: chains of FOLD l in acc, their sums over kFoldStages stages in mid, and
// those in sum, for contiguous fibres with what the additions round off in err. One chain of n_q would be
// further off than the eight chains of the column kernel or the chains of 32 of the l-split kernels
// (relative error at n_q = 1027: 1.0e-15 against 1.9e-16, 1.6e-16 with FOLD).
constexpr int kFoldStages = 8;

// One stage (16 l) of a warp's 16 rows x 8 N columns. At most eight columns: two accumulation
// chains (even and odd l / 4), added by the caller. FOLD: new chains, one or two of a stage.
template <int N, bool AK, bool BCM, int FOLD, int AR, int AP, int BR, int BP, int NA>
__device__ __forceinline__ void stage(const double (&sa)[AR][AP], const double (&sb)[BR][BP], int warp, int g, int c,
                                      double (&acc)[2][NA][2])
{
    if constexpr (N <= NA) {
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            // rows of mma r, group g: 2 g + r (strided fibres: one 16-byte load), 8 r + g otherwise
            double a0, a1;
            if (AK) {
                a0 = sa[warp * 16 + g][kk + c];
                a1 = sa[warp * 16 + 8 + g][kk + c];
            } else {
                const double2 t = *reinterpret_cast<const double2*>(&sa[kk + c][warp * 16 + 2 * g]);
                a0 = t.x;
                a1 = t.y;
            }
#pragma unroll
            for (int f = 0; f < N; ++f) {
                const double b = BCM ? sb[kk + c][8 * f + g] : sb[8 * f + g][kk + c];
                const int to = N == 1 ? (kk >> 2) & 1 : FOLD == 8 ? f + kk / 8 * N : f;
                if (FOLD && (N == 1 ? kk < 8 : kk % (FOLD ? FOLD : BK) == 0)) {
                    mma_open(acc[0][to], a0, b);
                    mma_open(acc[1][to], a1, b);
                } else {
                    mma(acc[0][to], a0, b);
                    mma(acc[1][to], a1, b);
                }
            }
        }
    }
}

// Tiles first, first + step, ... below `last`, l in [l_begin, l_end) of each; the stages of
// consecutive tiles follow one another through the ring, so that the next tile's loads are in
// flight while this one's results are stored. VEC: 16-byte copies of A (alignment checked by the
// host). The caller synchronises the block between two calls that share `sm`.
template <int BM, int NF, int ST, bool AK, bool VEC, bool BCM, bool EXACT, int FOLD>
__device__ __forceinline__ void tiles(const View3& v, int64_t first, int64_t step, int64_t last, const ColumnGrid& gr,
                                      Smem<BM, NF, ST, AK, BCM>& sm, int64_t l_begin, int64_t l_end)
{
    constexpr int BN = NF * 8, NT = 2 * BM, NA = NF == 1 || FOLD == 8 ? 2 * NF : NF;
    constexpr int SETS = FOLD == 8 || NF == 1 ? 2 : 1;   // chains of an output in a stage
    constexpr int NM = FOLD ? NF : 1;
    static_assert(!FOLD || (EXACT && NF <= 2 && BK % FOLD == 0), "folded builds are narrow and of one width");
    const double* __restrict__ A = static_cast<const double*>(v.a);
    const double* __restrict__ B = static_cast<const double*>(v.b);
    double* __restrict__ C = static_cast<double*>(v.c);
    const int64_t inner = v.inner, m = v.m, nq = v.nq;
    const int64_t M = v.outer * inner;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;

    // A copies: WA elements each, LA of them per thread and stage. Strided fibres: all of a
    // thread's copies are of the same rows, l apart; contiguous fibres: same l, rows apart.
    constexpr int WA = VEC ? 2 : 1, LA = BM * BK / WA / NT;
    constexpr int AX = (AK ? BK : BM) / WA;          // copies along the contiguous extent
    constexpr int AY = NT / AX;                      // rows of copies per pass
    static_assert(AX <= NT && AX * WA == (AK ? BK : BM) && AY * LA == (AK ? BM : BK), "the copies of a stage cover the tile exactly");
    const int ax = (tid % AX) * WA, ay = tid / AX;
    // B copies: 8 bytes each (any alignment of m and n_q), of the columns below 8 nf only
    constexpr int BX = !BCM ? BK : NF == 1 ? 8 : NF == 2 ? 16 : NF <= 4 ? 32 : 64, BY = NT / BX;
    constexpr int LB = ((BCM ? BK : BN) + BY - 1) / BY;
    const int bx = tid % BX, by = tid / BX;

    // the tile being loaded: this thread's first element of A and of B at the current stage, and
    // how much of the l range is left
    int64_t lt = first, left = 0;
    int a_rows = 0;          // rows of the tile in A
    int64_t b_cols = 0;      // columns of B from this tile's first
    const double* ap = A;
    const double* bp = B;
    auto start = [&]() {
        const int64_t rt = gr.cols == 1 ? lt : slice_of(lt, gr.cols);
        const int64_t m0 = rt * BM, n0 = (lt - rt * gr.cols) * gr.nf * 8;
        left = l_end - l_begin;
        b_cols = m - n0;
        if (!EXACT && b_cols > gr.nf * 8) b_cols = gr.nf * 8;
        a_rows = (int)(M - m0 < BM ? M - m0 : BM);
        if (AK) {
            ap = A + (m0 + ay) * nq + l_begin + ax;
        } else {
            const int64_t row = m0 + ax, k = slice_of(row, inner);
            ap = A + (k * nq + l_begin + ay) * inner + (row - k * inner);
        }
        bp = BCM ? B + (l_begin + by) * m + n0 + bx : B + (n0 + by) * nq + l_begin + bx;
    };
    // copies with !ok zero their destination and read nothing (their addresses may lie outside)
    const int64_t a_step = AK ? (int64_t)AY * nq : (int64_t)AY * inner, b_step = BCM ? BY * m : BY * nq;
    auto issue = [&](int st) {
        const int n = left < BK ? (int)left : BK;
#pragma unroll
        for (int s = 0; s < LA; ++s) {
            const int yo = ay + s * AY;   // [row][l] or [l][row]
            const bool ok = AK ? yo < a_rows && ax < n : ax < a_rows && yo < n;
            if (VEC) copy16(&sm.a[st][yo][ax], ap + s * a_step, ok);
            else copy8(&sm.a[st][yo][ax], ap + s * a_step, ok);
        }
#pragma unroll
        for (int s = 0; s < LB; ++s) {
            const int jo = BCM ? bx : by + s * BY, lo = BCM ? by + s * BY : bx;
            if (jo >= BN || lo >= BK) continue;
            copy8(BCM ? &sm.b[st][lo][jo] : &sm.b[st][jo][lo], bp + s * b_step, jo < b_cols && lo < n);
        }
    };
    // loads one stage (none past the last tile) and moves on; one commit group per call, empty
    // ones too, so that wait_group counts stages
    auto load_next = [&](int st) {
        if (lt < last) {
            issue(st);
            left -= BK;
            ap += AK ? BK : BK * inner;
            bp += BCM ? BK * m : BK;
            if (left <= 0) {
                lt += step;
                if (lt < last) start();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (lt < last) start();
#pragma unroll
    for (int st = 0; st < ST - 1; ++st) load_next(st);
    int rd = 0, wr = ST - 1;
    const int nk = (int)ceil_div(l_end - l_begin, BK);

    for (int64_t t = first; t < last; t += step) {
    const int64_t t_row = gr.cols == 1 ? t : slice_of(t, gr.cols);
    const int64_t m0 = t_row * BM, n0 = (t - t_row * gr.cols) * gr.nf * 8;
    const int nf = EXACT ? NF : (int)(m - n0 < gr.nf * 8 ? (m - n0 + 7) / 8 : gr.nf);

    double acc[2][NA][2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int f = 0; f < NA; ++f) acc[r][f][0] = acc[r][f][1] = 0.0;
    double mid[2][NM][2], sum[2][NM][2], err[2][NM][2];
    // the last stage's chains into mid. Called once the next stage's copies are on their way: right after
    // the stage the additions would wait for its last mma (43 us against 37 at 4096 rows, n_q = 4096, m = 16)
    auto close_chains = [&]() {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int f = 0; f < NM; ++f)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    mid[r][f][e] += SETS == 2 ? acc[r][f][e] + acc[r][f + NF < NA ? f + NF : 0][e] : acc[r][f][e];
    };
    auto fold = [&]() {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int f = 0; f < NM; ++f)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (AK) add_kept(sum[r][f][e], err[r][f][e], mid[r][f][e]);
                    else sum[r][f][e] += mid[r][f][e];
                    mid[r][f][e] = 0.0;
                }
    };
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int f = 0; f < NM; ++f)
#pragma unroll
            for (int e = 0; e < 2; ++e) mid[r][f][e] = sum[r][f][e] = err[r][f][e] = 0.0;

    // stage rd has landed for all, and all have read stage wr's last contents (a warp at a time reaches
    // this barrier from one of the two loops below)
    auto turn = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        asm volatile("bar.sync 0;" ::: "memory");
        load_next(wr);
    };
    auto advance = [&]() {
        rd = rd + 1 == ST ? 0 : rd + 1;
        wr = wr + 1 == ST ? 0 : wr + 1;
    };
    const int mine = m0 + warp * 16 < M ? nk : 0;   // a warp past the last row only copies
    for (int kt = mine; kt < nk; ++kt) {
        turn();
        advance();
    }
    for (int kt = 0; kt < mine; ++kt) {
        turn();
        if constexpr (EXACT) {
            if constexpr (FOLD != 0) {
                if (kt > 0) close_chains();
                if (kt % kFoldStages == 0) fold();
            }
            stage<NF, AK, BCM, FOLD>(sm.a[rd], sm.b[rd], warp, g, c, acc);
        } else {
            // one build per width: predicated-off mma would take the pipe as long as executed ones
            switch (nf) {
            case 1: stage<1, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 2: stage<2, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 3: stage<3, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 4: stage<4, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 5: stage<5, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 6: stage<6, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            case 7: stage<7, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            default: stage<NF, AK, BCM, 0>(sm.a[rd], sm.b[rd], warp, g, c, acc); break;
            }
        }
        advance();
    }

    if constexpr (FOLD != 0) {
        close_chains();
        fold();
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int f = 0; f < NM; ++f)
#pragma unroll
                for (int e = 0; e < 2; ++e) acc[r][f][e] = AK ? kept_total(sum[r][f][e], err[r][f][e]) : sum[r][f][e];
    } else if (nf == 1) {
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[r][0][e] += acc[r][1][e];
    }

    // C(row, j) = base(row) + j inner; lane (g, c) holds columns 8 f + 2 c and 8 f + 2 c + 1
    const bool c16 = (reinterpret_cast<uintptr_t>(C) & 15u) == 0;
    if (AK) {
        const bool vec = c16 && (m & 1) == 0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t row = m0 + warp * 16 + 8 * r + g;
            if (row >= M) continue;
            double* cp = C + row * m;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const int64_t j = n0 + 8 * f + 2 * c;
                if (f >= nf || j >= m) continue;
                if (vec) {
                    *reinterpret_cast<double2*>(cp + j) = make_double2(acc[r][f][0], acc[r][f][1]);
                } else {
                    cp[j] = acc[r][f][0];
                    if (j + 1 < m) cp[j + 1] = acc[r][f][1];
                }
            }
        }
    } else {
        const int64_t row = m0 + warp * 16 + 2 * g;
        if (row >= M) continue;
        const int64_t k0 = slice_of(row, inner), i0 = row - k0 * inner;
        double* cp = C + k0 * inner * m + i0;
        if (c16 && (inner & 1) == 0) {
            // row + 1 lies in the same slice (and M is even)
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t j = n0 + 8 * f + 2 * c + e;
                    if (f < nf && j < m)
                        *reinterpret_cast<double2*>(cp + j * inner) = make_double2(acc[0][f][e], acc[1][f][e]);
                }
        } else {
            const bool two = row + 1 < M;
            // the next row: i + 1 of this slice, or i = 0 of the next
            double* cq = i0 + 1 < inner ? cp + 1 : C + (k0 + 1) * inner * m;
#pragma unroll
            for (int f = 0; f < NF; ++f)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int64_t j = n0 + 8 * f + 2 * c + e;
                    if (f < nf && j < m) {
                        cp[j * inner] = acc[0][f][e];
                        if (two) cq[j * inner] = acc[1][f][e];
                    }
                }
        }
    }
    }
}

}  // namespace f64
}  // namespace tlibttm
