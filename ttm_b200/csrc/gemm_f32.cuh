// FP32 slice-GEMM on packed FFMA pairs: every output is one chain of correctly rounded fused
// multiply-adds in the order of l (tiles of 128 rows and at most 16 columns: chains of eight, added up in
// two more levels).
//
// One tile is 32 TM rows (flattened (k, i) pairs) x TX TN columns j; 32 x TX threads (TX 8 or 4), each
// TM x TN outputs. Accumulators pair neighbouring rows, which come from shared memory as 64-bit
// halves of a 16-byte load; each column value is duplicated once for TM / 2 pairs. Widths are whole
// builds in groups of eight columns, so that padding of m is not multiplied (m = 100: two tiles of
// 56). A warp is 8 x 4 threads (4 x 8 for wide tiles of contiguous fibres): its 16-byte loads of A and B cover
// at most 128 distinct bytes (one wavefront each), its stores of C 128 contiguous bytes.
// A and B tiles of 16 l go through a ring of ST shared-memory stages filled with cp.async, B as
// [l][j], A as [l][row] for rows of i and as [row][l] for contiguous fibres (whose accumulators pair
// neighbouring columns instead).
//
// What bounds it: the FMA pipe (73.7 TFLOP/s for a stream of packed FFMA; the inner loop of 8 x 8
// outputs alone runs at 63-66) from m about 24 on, below that shared-memory reads and then reading A.
// The loads of a stage must be cheap next to its 512 packed FMA a thread: running pointers instead of
// addresses recomputed per copy gave 46.8 -> 53 TFLOP/s. Measured against the register-staged 128 x
// 128 tile before it: A 32^2 x 64 x 32^2, mode of 64, m = 64 468 -> 190 us; A 2^26, n_q = 256, m = 64
// 423 -> 168 us, m = 512 1706 -> 1300 us; contiguous fibres of 64, m = 64 426 -> 239 us; m = 17,
// fibres of 40, 363 -> 77 us. Contiguous fibres keep to 45 TFLOP/s (the wide build spills a little).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace tlibttm {
namespace f32 {

constexpr int BK = 16;

template <int TX, int TM, int TN, int ST, bool AK>
struct Smem {
    static constexpr int BM = 32 * TM, BN = TX * TN;
    static constexpr int AP = AK ? BK + 4 : BM + 4, AR = AK ? BM : BK, BP = (BN + 31) / 32 * 32 + 4;
    __align__(16) float a[ST][AR][AP];   // [row][l] for contiguous fibres, else [l][row]
    __align__(16) float b[ST][BK][BP];
};

__device__ __forceinline__ void copy16(void* dst, const void* src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy4(void* dst, const void* src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}

// Column q of a thread's TN: chunks of four columns 4 TX apart, then one of two and one of one.
template <int TX, int TN>
__device__ __forceinline__ int column(int q, int tx)
{
    constexpr int F = TN / 4 * 4;   // columns in chunks of four
    if (q < F) return q / 4 * 4 * TX + tx * 4 + q % 4;
    if ((TN & 2) && q < F + 2) return F * TX + tx * 2 + (q - F);
    return (TN & ~1) * TX + tx;
}

// The thread's TN column values of one l.
template <int TX, int TN, int BP>
__device__ __forceinline__ void load_columns(float (&b)[TN], const float (&sb)[BP], int tx)
{
    constexpr int F = TN / 4 * 4;
#pragma unroll
    for (int q = 0; q < F; q += 4) {
        const float4 t = *reinterpret_cast<const float4*>(&sb[column<TX, TN>(q, tx)]);
        b[q] = t.x;
        b[q + 1] = t.y;
        b[q + 2] = t.z;
        b[q + 3] = t.w;
    }
    if constexpr (TN & 2) {
        const float2 t = *reinterpret_cast<const float2*>(&sb[column<TX, TN>(F, tx)]);
        b[F] = t.x;
        b[F + 1] = t.y;
    }
    if constexpr (TN & 1) b[TN - 1] = sb[column<TX, TN>(TN - 1, tx)];
}

// Tiles of 128 rows and at most 16 columns (FOLD) add up in levels: chains of kFoldChain l in acc, their sums over
// kFoldStages stages in mid, and those in sum with what the additions round off in err. The kernels that
// they take problems from add up in several shorter chains (eight, or chains of 32 in the l-split
// kernels), which one chain of n_q would be further off than. Relative error against FP64, N(0,1)
// entries: one chain 1.4e-7 at n_q = 64, 5.7e-7 at 1024, 1.6e-6 at 8000; the kernels replaced 0.8e-7
// to 4.1e-7; these levels 0.8e-7 to 1.0e-7 at any n_q. They want 128 registers: at 96 (five blocks
// an SM) they took 37 us on 4096 rows of i, n_q = 1024, m = 16 in place of 31 (one chain: 29).
constexpr int kFoldChain = 8, kFoldStages = 8;

// A thread's outputs where rows of i are contiguous: acc[p][q] holds rows 2 p and 2 p + 1 of its TM
// (chunks of four rows 128 apart), column q.
template <int TX, int TM, int NA, bool FOLD, bool HALF>
struct AccRows {
    unsigned long long acc[TM / 2][NA];
    static constexpr int FP = FOLD ? TM / 2 : 1, FQ = FOLD ? NA : 1;
    unsigned long long mid[FP][FQ], sum[FP][FQ], err[FP][FQ];

    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int p = 0; p < TM / 2; ++p)
#pragma unroll
            for (int q = 0; q < NA; ++q) {
                acc[p][q] = 0ull;
                if constexpr (FOLD) mid[p][q] = sum[p][q] = err[p][q] = 0ull;
            }
    }

    // FOLD: the sum of kFoldStages stages goes into the total
    __device__ __forceinline__ void fold()
    {
#pragma unroll
        for (int p = 0; p < TM / 2; ++p)
#pragma unroll
            for (int q = 0; q < NA; ++q) {
                add_kept(sum[p][q], err[p][q], mid[p][q]);
                mid[p][q] = 0ull;
            }
    }

    __device__ __forceinline__ void finish()
    {
#pragma unroll
        for (int p = 0; p < TM / 2; ++p)
#pragma unroll
            for (int q = 0; q < NA; ++q) {
                add_kept(sum[p][q], err[p][q], mid[p][q]);
                acc[p][q] = kept_total(sum[p][q], err[p][q]);
            }
    }

    // one stage: 16 l, with HALF only its first 8 where n, those left of the range, are no more
    template <int TN, int AP, int BP>
    __device__ __forceinline__ void stage(const float (&sa)[BK][AP], const float (&sb)[BK][BP], int ty, int tx, int n)
    {
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            if (HALF && kk == BK / 2 && n <= BK / 2) break;   // the rest is padding
            unsigned long long a[TM / 2], bq[TN];
#pragma unroll
            for (int h = 0; h < TM / 4; ++h) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&sa[kk][h * 128 + ty * 4]);
                a[2 * h] = t.x;
                a[2 * h + 1] = t.y;
            }
            float b[TN];
            load_columns<TX, TN>(b, sb[kk], tx);
#pragma unroll
            for (int q = 0; q < TN; ++q) bq[q] = pair_dup(b[q]);
#pragma unroll
            for (int p = 0; p < TM / 2; ++p)
#pragma unroll
                for (int q = 0; q < TN; ++q) {
                    if (FOLD && kk % kFoldChain == 0) acc[p][q] = mul2(a[p], bq[q]);
                    else ffma2(acc[p][q], a[p], bq[q]);
                    if constexpr (FOLD)
                        if (kk % kFoldChain == kFoldChain - 1) mid[p][q] = add2(mid[p][q], acc[p][q]);
                }
        }
    }

    template <int TN>
    __device__ __forceinline__ void store(const View3& v, int64_t m0, int64_t n0, int ty, int tx) const
    {
        float* __restrict__ C = static_cast<float*>(v.c);
        const int64_t inner = v.inner, m = v.m, M = v.outer * inner;
        const bool vec = (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && inner % 4 == 0;
#pragma unroll
        for (int h = 0; h < TM / 4; ++h) {
            const int64_t row0 = m0 + h * 128 + ty * 4;
            if (row0 >= M) continue;
            int64_t k = slice_of(row0, inner), i = row0 - k * inner;
            float* cp = C + k * inner * m + i;
            if (vec) {
                // the four rows lie in one slice (and M is a multiple of four)
#pragma unroll
                for (int q = 0; q < TN; ++q) {
                    const int64_t j = n0 + column<TX, TN>(q, tx);
                    if (j < m)
                        *reinterpret_cast<float4*>(cp + j * inner) =
                            make_float4(pair_lo(acc[2 * h][q]), pair_hi(acc[2 * h][q]), pair_lo(acc[2 * h + 1][q]),
                                        pair_hi(acc[2 * h + 1][q]));
                }
                continue;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (row0 + r < M) {
#pragma unroll
                    for (int q = 0; q < TN; ++q) {
                        const int64_t j = n0 + column<TX, TN>(q, tx);
                        const unsigned long long x = acc[2 * h + r / 2][q];
                        if (j < m) cp[j * inner] = r & 1 ? pair_hi(x) : pair_lo(x);
                    }
                }
                // the next row: i + 1 of this slice, or i = 0 of the next
                if (++i < inner) ++cp;
                else {
                    i = 0;
                    cp = C + ++k * inner * m;
                }
            }
        }
    }
};

// A thread's outputs where fibres are contiguous: rows 32 apart, acc[r][p] holds columns 2 p and
// 2 p + 1 of row r, last[r] the column left over. A's rows come four l at a time.
template <int TX, int TM, int NA, bool FOLD, bool HALF>
struct AccFibres {
    static constexpr int NP = NA / 2;   // column pairs
    unsigned long long acc[TM][NP > 0 ? NP : 1];
    float last[TM];
    static constexpr int FR = FOLD ? TM : 1;
    unsigned long long mid[FR][NP > 0 ? NP : 1], sum[FR][NP > 0 ? NP : 1], err[FR][NP > 0 ? NP : 1];
    float mid_last[FR], sum_last[FR], err_last[FR];

    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int r = 0; r < TM; ++r) {
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                acc[r][p] = 0ull;
                if constexpr (FOLD) mid[r][p] = sum[r][p] = err[r][p] = 0ull;
            }
            last[r] = 0.0f;
            if constexpr (FOLD) mid_last[r] = sum_last[r] = err_last[r] = 0.0f;
        }
    }

    __device__ __forceinline__ void fold()
    {
#pragma unroll
        for (int r = 0; r < TM; ++r) {
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                add_kept(sum[r][p], err[r][p], mid[r][p]);
                mid[r][p] = 0ull;
            }
            add_kept(sum_last[r], err_last[r], mid_last[r]);
            mid_last[r] = 0.0f;
        }
    }

    __device__ __forceinline__ void finish()
    {
#pragma unroll
        for (int r = 0; r < TM; ++r) {
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                add_kept(sum[r][p], err[r][p], mid[r][p]);
                acc[r][p] = kept_total(sum[r][p], err[r][p]);
            }
            add_kept(sum_last[r], err_last[r], mid_last[r]);
            last[r] = kept_total(sum_last[r], err_last[r]);
        }
    }

    template <int TN, int AR, int AP, int BP>
    __device__ __forceinline__ void stage(const float (&sa)[AR][AP], const float (&sb)[BK][BP], int ty, int tx, int n)
    {
#pragma unroll
        for (int k2 = 0; k2 < BK; k2 += 2) {
            if (HALF && k2 == BK / 2 && n <= BK / 2) break;
            float2 a[TM];
#pragma unroll
            for (int r = 0; r < TM; ++r) a[r] = *reinterpret_cast<const float2*>(&sa[r * 32 + ty][k2]);
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                float b[TN];
                load_columns<TX, TN>(b, sb[k2 + kk], tx);
#pragma unroll
                for (int r = 0; r < TM; ++r) {
                    const float x = kk == 0 ? a[r].x : a[r].y;
                    const unsigned long long xx = pair_dup(x);
                    const bool open = FOLD && (k2 + kk) % kFoldChain == 0;
                    const bool close = FOLD && (k2 + kk) % kFoldChain == kFoldChain - 1;
#pragma unroll
                    for (int p = 0; p < TN / 2; ++p) {
                        const unsigned long long bp = pair_of(b[2 * p], b[2 * p + 1]);
                        if (open) acc[r][p] = mul2(xx, bp);
                        else ffma2(acc[r][p], xx, bp);
                        if constexpr (FOLD)
                            if (close) mid[r][p] = add2(mid[r][p], acc[r][p]);
                    }
                    if constexpr (TN & 1) {
                        last[r] = open ? __fmul_rn(x, b[TN - 1]) : __fmaf_rn(x, b[TN - 1], last[r]);
                        if constexpr (FOLD)
                            if (close) mid_last[r] = __fadd_rn(mid_last[r], last[r]);
                    }
                }
            }
        }
    }

    template <int TN>
    __device__ __forceinline__ void store(const View3& v, int64_t m0, int64_t n0, int ty, int tx) const
    {
        float* __restrict__ C = static_cast<float*>(v.c);
        const int64_t m = v.m, M = v.outer;
        const bool vec = (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && m % 4 == 0;
#pragma unroll
        for (int r = 0; r < TM; ++r) {
            const int64_t row = m0 + r * 32 + ty;
            if (row >= M) continue;
            float* cp = C + row * m;
            float x[TN];
#pragma unroll
            for (int q = 0; q < TN; ++q)
                x[q] = q == TN - 1 && (TN & 1) ? last[r] : q & 1 ? pair_hi(acc[r][q / 2]) : pair_lo(acc[r][q / 2]);
#pragma unroll
            for (int q = 0; q < TN; ++q) {
                const int64_t j = n0 + column<TX, TN>(q, tx);
                if (vec && q < TN / 4 * 4) {
                    if (q % 4 == 0 && j < m)
                        *reinterpret_cast<float4*>(cp + j) = make_float4(x[q], x[q + 1], x[q + 2], x[q + 3]);
                } else if (j < m) {
                    cp[j] = x[q];
                }
            }
        }
    }
};

// Tiles first, first + step, ... below `last`, l in [l_begin, l_end) of each; the stages of
// consecutive tiles follow one another through the ring. VEC: 16-byte copies of A (alignment
// checked by the host). EXACT: every tile has TN groups of columns, else gr.nf <= TN. HALF: a last
// stage of at most 8 l multiplies 8 (a branch in every stage, which costs long ranges up to 9 %).
// The caller synchronises the block between two calls that share `sm`.
template <int TX, int TM, int TN, int ST, bool AK, bool VEC, bool BCM, bool EXACT, bool HALF = false>
__device__ __forceinline__ void tiles(const View3& v, int64_t first, int64_t step, int64_t last, const ColumnGrid& gr,
                                      Smem<TX, TM, TN, ST, AK>& sm, int64_t l_begin, int64_t l_end)
{
    constexpr int BM = 32 * TM, BN = TX * TN, NT = 32 * TX;
    constexpr bool FOLD = TM == 4 && TX * TN <= 16;
    static_assert(!FOLD || EXACT, "the narrower widths of an inexact build are not folded");
    const float* __restrict__ A = static_cast<const float*>(v.a);
    const float* __restrict__ B = static_cast<const float*>(v.b);
    const int64_t inner = v.inner, m = v.m, nq = v.nq;
    const int64_t M = v.outer * inner;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // rows of i: 8 x 4 threads a warp; contiguous fibres 4 x 8 where there are eight along the columns, so
    // that a store of C covers whole lines
    constexpr bool LINES = AK && TX == 8;
    const int ty = LINES ? warp * 4 + (lane >> 3) : warp / (TX / 4) * 8 + (lane & 7);
    const int tx = LINES ? lane & 7 : warp % (TX / 4) * 4 + (lane >> 3);

    // A copies of WA elements: AX along the contiguous extent (l or the rows), AY of the other per pass
    // (an extent longer than the block takes RP parts of NT copies each)
    constexpr int WA = VEC ? 4 : 1;
    constexpr int AE = (AK ? BK : BM) / WA, AX = AE < NT ? AE : NT, AY = NT / AX, RP = AE / AX;
    constexpr int LA = (AK ? BM : BK) / AY;
    static_assert(AX * RP * WA == (AK ? BK : BM) && AY * LA == (AK ? BM : BK) && (!AK || RP == 1),
                  "the copies of a stage cover the tile exactly");
    const int ax = (tid % AX) * WA, ay = tid / AX;
    // B copies: one element each, of the columns below the tile's width
    constexpr int BX = !BCM ? 8 : BN <= 8 ? 8 : BN <= 16 ? 16 : BN <= 32 ? 32 : 64, BY = NT / BX;
    const int bx = tid % BX, by = tid / BX;
    constexpr int LB = BCM ? (BK + BY - 1) / BY : 2 * ((BN + BY - 1) / BY);

    // the tile being loaded: this thread's first element of A and of B at the current stage, and
    // how much of the l range is left
    int64_t lt = first, left = 0;
    int a_rows = 0;          // rows of the tile in A
    int64_t b_cols = 0;      // columns of B from this tile's first
    const float* ap[RP];
    const float* bp = B;
    auto start = [&]() {
        const int64_t rt = gr.cols == 1 ? lt : slice_of(lt, gr.cols);
        const int64_t m0 = rt * BM, n0 = (lt - rt * gr.cols) * gr.nf * TX;
        left = l_end - l_begin;
        b_cols = m - n0;
        if (!EXACT && b_cols > gr.nf * TX) b_cols = gr.nf * TX;
        a_rows = (int)(M - m0 < BM ? M - m0 : BM);
#pragma unroll
        for (int h = 0; h < RP; ++h) {
            if (AK) {
                ap[h] = A + (m0 + ay) * nq + l_begin + ax;
            } else {
                const int64_t row = m0 + ax + h * NT * WA, k = slice_of(row, inner);
                ap[h] = A + (k * nq + l_begin + ay) * inner + (row - k * inner);
            }
        }
        bp = BCM ? B + (l_begin + by) * m + n0 + bx : B + (n0 + by) * nq + l_begin + bx;
    };
    // copies with !ok zero their destination and read nothing (their addresses may lie outside)
    const int64_t a_step = AK ? (int64_t)AY * nq : (int64_t)AY * inner, b_step = BCM ? BY * m : BY * nq;
    auto issue = [&](int st) {
        const int n = left < BK ? (int)left : BK;
#pragma unroll
        for (int h = 0; h < RP; ++h)
#pragma unroll
            for (int s = 0; s < LA; ++s) {
                const int yo = ay + s * AY, xo = ax + h * NT * WA;   // [row][l] or [l][row]
                const bool ok = AK ? yo < a_rows && xo < n : xo < a_rows && yo < n;
                if (VEC) copy16(&sm.a[st][yo][xo], ap[h] + s * a_step, ok);
                else copy4(&sm.a[st][yo][xo], ap[h] + s * a_step, ok);
            }
#pragma unroll
        for (int s = 0; s < LB; ++s) {
            const int jo = BCM ? bx : by + (s >> 1) * BY, lo = BCM ? by + s * BY : bx + (s & 1) * 8;
            if (jo >= BN || lo >= BK) continue;
            copy4(&sm.b[st][lo][jo], BCM ? bp + s * b_step : bp + (s >> 1) * b_step + (s & 1) * 8, jo < b_cols && lo < n);
        }
    };
    // loads one stage (none past the last tile) and moves on; one commit group per call, empty
    // ones too, so that wait_group counts stages
    auto load_next = [&](int st) {
        if (lt < last) {
            issue(st);
            left -= BK;
#pragma unroll
            for (int h = 0; h < RP; ++h) ap[h] += AK ? BK : BK * inner;
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
        typename std::conditional<AK, AccFibres<TX, TM, TN, FOLD, HALF>, AccRows<TX, TM, TN, FOLD, HALF>>::type out;
        out.clear();
        for (int kt = 0; kt < nk; ++kt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncthreads();   // stage rd has landed for all, and all have read stage wr's last contents
            load_next(wr);
            if constexpr (EXACT) {
                out.template stage<TN>(sm.a[rd], sm.b[rd], ty, tx, (int)(l_end - l_begin) - kt * BK);
                if constexpr (FOLD)
                    if (kt % kFoldStages == kFoldStages - 1) out.fold();
            } else {
                if (gr.nf > 6) out.template stage<TN>(sm.a[rd], sm.b[rd], ty, tx, (int)(l_end - l_begin) - kt * BK);
                else if (gr.nf > 4) out.template stage<6>(sm.a[rd], sm.b[rd], ty, tx, (int)(l_end - l_begin) - kt * BK);
                else out.template stage<4>(sm.a[rd], sm.b[rd], ty, tx, (int)(l_end - l_begin) - kt * BK);
            }
            rd = rd + 1 == ST ? 0 : rd + 1;
            wr = wr + 1 == ST ? 0 : wr + 1;
        }
        if constexpr (FOLD) out.finish();
        const int64_t rt = gr.cols == 1 ? t : slice_of(t, gr.cols);
        const int64_t n0 = (t - rt * gr.cols) * gr.nf * TX;
        if constexpr (EXACT) {
            out.template store<TN>(v, rt * BM, n0, ty, tx);
        } else {
            if (gr.nf > 6) out.template store<TN>(v, rt * BM, n0, ty, tx);
            else if (gr.nf > 4) out.template store<6>(v, rt * BM, n0, ty, tx);
            else out.template store<4>(v, rt * BM, n0, ty, tx);
        }
    }
}

}  // namespace f32
}  // namespace tlibttm
