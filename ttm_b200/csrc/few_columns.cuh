// FP32 small-m kernel (m <= 8) for rows of i whose lines are not on 16-byte boundaries (inner % 4 != 0,
// A itself on one): exact FMA, C(k, j, i) = sum_l A(k, l, i) B(j, l).
//
// A tile is 256 consecutive i of one slice; 128 threads. Each line (k, l) of the tile is copied 16
// bytes at a time from the boundary at or below its first element and so starts 0 to 3 elements into
// its line in shared memory; a line's last copy stops at its end, so that only the elements before a
// line in its first 16 bytes are read besides it. Lane t holds rows t, t + 32, ... of the tile, so that
// shared-memory reads hit 32 banks whatever the shift, and all TN columns; the four warps take every
// fourth l, and their sums are added in a fixed order at the end. Where the column kernel would add up in
// eight chains per output, one chain per warp was further off (1.9e-7 against 1.4e-7 at n_q = 400,
// relative to FP64): a warp's l are cut into chains of 8, or 16 from n_q = 128 on (1.0e-7), at 15 or 8 %
// of the time at m = 8.
//
// What bounds it: reading A. The column kernel's copies of one element per lane (colvec_async) took
// 12 cycles an instruction and SM and held it to 2.7-3.1 TB/s; the slice-GEMM tile reads each
// element of A from shared memory four times. The copies bypass L1 (through it, 28 KB of which the
// rings leave, they took 64 us instead of 45 at m = 4). Measured on A (401, 263, 509), middle mode:
// m = 1 71 -> 41 us, m = 4 73 -> 45, m = 7 83 -> 51 (4.3 TB/s).
#pragma once

#include "common.cuh"

namespace tlibttm {
namespace few {

constexpr int BM = 256, BK = 16, NT = 128, ST = 3, WARPS = NT / 32, RPL = BM / 32;

template <int TN>
struct Smem {
    __align__(16) float a[ST][BK][BM + 4];
    __align__(16) float b[ST][BK][TN];
    float red[WARPS][TN < 4 ? TN : 4][BM];
};

// Copies the first `bytes` (0 to 16) of 16 aligned bytes and zeroes the rest.
__device__ __forceinline__ void copy16_part(void* dst, const void* src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy4(void* dst, const void* src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(ok ? 4 : 0)
                 : "memory");
}

// Tile `t` of outer * ceil(inner / 256). CHAINS: a warp's chains are `chain` + 1 stages (a power of two) of
// four l of its own; else it has one.
template <int TN, bool BCM, bool CHAINS>
__device__ __forceinline__ void tile(const View3& v, int64_t t, int chain, Smem<TN>& sm)
{
    const float* __restrict__ A = static_cast<const float*>(v.a);
    const float* __restrict__ B = static_cast<const float*>(v.b);
    const int64_t inner = v.inner, nq = v.nq, per_slice = (inner + BM - 1) / BM;
    const int m = (int)v.m;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t k = slice_of(t, per_slice), i0 = (t - k * per_slice) * BM;
    const int rows = (int)(inner - i0 < BM ? inner - i0 : BM);
    // lines: 64 copies of 16 bytes each, two lines per pass of the block, and one copy more
    constexpr int CX = BM / 4, CY = NT / CX;
    static_assert(CX * CY == NT && BK % CY == 0 && BK <= NT && BK * TN <= NT, "the copies of a stage cover it exactly");
    const int cx = tid % CX * 4, cy = tid / CX;
    const int bj = BCM ? tid % TN : tid / BK, bl = BCM ? tid / TN : tid % BK;
    const float* bp = BCM ? B + (int64_t)bl * m + bj : B + (int64_t)bj * nq + bl;
    int64_t line0 = k * nq * inner + i0, left = nq;   // the stage being loaded
    auto load_next = [&](int st) {
        if (left > 0) {
            const int n = left < BK ? (int)left : BK;
            auto line_copy = [&](int y, int x) {
                const int64_t at = line0 + y * inner;
                const int have = y < n ? (int)(at & 3) + rows - x : 0;   // elements of the line from here on
                copy16_part(&sm.a[st][y][x], A + (at & ~int64_t(3)) + x, have <= 0 ? 0 : have >= 4 ? 16 : have * 4);
            };
#pragma unroll
            for (int s = 0; s < BK / CY; ++s) line_copy(cy + s * CY, cx);
            if (tid < BK) line_copy(tid, BM);
            if (tid < BK * TN) copy4(&sm.b[st][bl][bj], bp, bj < m && bl < n);
            line0 += BK * inner;
            bp += BCM ? (int64_t)BK * m : BK;
            left -= BK;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");   // one per stage, empty ones too
    };
#pragma unroll
    for (int st = 0; st < ST - 1; ++st) load_next(st);

    // this warp's l (warp, warp + 4, ...) all have one residue mod 4, and so one shift: BK inner and
    // BM are multiples of four
    const int sh = (int)((((uint32_t)k * (uint32_t)nq + (uint32_t)warp) * (uint32_t)inner) & 3u);
    unsigned long long acc[RPL / 2][TN], sum[CHAINS ? RPL / 2 : 1][TN];   // rows 64 p + lane and 64 p + 32 + lane
#pragma unroll
    for (int p = 0; p < RPL / 2; ++p)
#pragma unroll
        for (int q = 0; q < TN; ++q) {
            acc[p][q] = 0ull;
            if (CHAINS) sum[p][q] = 0ull;
        }
    int rd = 0, wr = ST - 1;
    const int nk = (int)ceil_div(nq, BK);
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();
        load_next(wr);
#pragma unroll
        for (int e = 0; e < BK / WARPS; ++e) {
            const int l = e * WARPS + warp;
            const float* ar = &sm.a[rd][l][lane + sh];
            unsigned long long a[RPL / 2];
#pragma unroll
            for (int p = 0; p < RPL / 2; ++p) a[p] = pair_of(ar[64 * p], ar[64 * p + 32]);
            float b[TN];
#pragma unroll
            for (int q = 0; q < TN; ++q) b[q] = sm.b[rd][l][q];
#pragma unroll
            for (int q = 0; q < TN; ++q) {
                const unsigned long long bq = pair_dup(b[q]);
#pragma unroll
                for (int p = 0; p < RPL / 2; ++p) ffma2(acc[p][q], a[p], bq);
            }
        }
        if (CHAINS && (kt & chain) == chain) {   // a chain ends
#pragma unroll
            for (int p = 0; p < RPL / 2; ++p)
#pragma unroll
                for (int q = 0; q < TN; ++q) {
                    sum[p][q] = add2(sum[p][q], acc[p][q]);
                    acc[p][q] = 0ull;
                }
        }
        rd = rd + 1 == ST ? 0 : rd + 1;
        wr = wr + 1 == ST ? 0 : wr + 1;
    }
    if (CHAINS) {
#pragma unroll
        for (int p = 0; p < RPL / 2; ++p)
#pragma unroll
            for (int q = 0; q < TN; ++q) acc[p][q] = add2(sum[p][q], acc[p][q]);
    }
    // the warps' sums, up to four columns at a time: thread t adds rows t and t + 128
    float* __restrict__ C = static_cast<float*>(v.c) + k * m * inner + i0;
    constexpr int QC = TN < 4 ? TN : 4;
#pragma unroll
    for (int q0 = 0; q0 < TN; q0 += QC) {
        if (q0 >= m) break;
        if (q0 > 0) __syncthreads();
#pragma unroll
        for (int q = 0; q < QC; ++q)
#pragma unroll
            for (int p = 0; p < RPL / 2; ++p) {
                sm.red[warp][q][64 * p + lane] = pair_lo(acc[p][q0 + q]);
                sm.red[warp][q][64 * p + 32 + lane] = pair_hi(acc[p][q0 + q]);
            }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < QC; ++q) {
            if (q0 + q >= m) break;
#pragma unroll
            for (int r = tid; r < BM; r += NT) {
                float s = sm.red[0][q][r];
#pragma unroll
                for (int w = 1; w < WARPS; ++w) s += sm.red[w][q][r];
                if (r < rows) C[(q0 + q) * inner + r] = s;
            }
        }
    }
}

}  // namespace few
}  // namespace tlibttm
