// SIMT kernels of the B200 TTM library: the exact-arithmetic ("plain") paths.
//
//  simt_gemm  slice-GEMM over the dense view C[k][j][i] = sum_l A[k][l][i] B(j,l):
//             FP32 on packed FFMA (gemm_f32.cuh), FP64 on the double-precision
//             matrix instruction (gemm_f64.cuh). Rows of the GEMM are the
//             flattened (k, i) pairs, so one kernel covers every layout case
//             without transposing anything.
//  colvec     bandwidth kernel for small m when A's fibres along mode q are
//             strided (inner >= 2): each thread owns W consecutive i of one k
//             and streams 16-byte loads along l; B is staged in shared memory.
//  rowdot     bandwidth kernel for small m when the fibres are contiguous
//             (inner == 1, q = pi_1): a group of G lanes reads one fibre with
//             16-byte loads and reduces the m partial sums by warp shuffles.
//  strided    definition-level kernel for non-dense (but valid) strides.
//
// All index arithmetic is 64-bit (a 256^4 tensor has 2^32 elements).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "few_columns.cuh"
#include "gemm_f32.cuh"
#include "gemm_f64.cuh"
#include "tc_kernels.cuh"

namespace tlibttm {
namespace {

template <typename T> struct V16;
template <> struct V16<float> { using type = float4; };
template <> struct V16<double> { using type = double2; };

template <typename T, int W>
__device__ __forceinline__ void load_vec(T (&r)[W], const T* p)
{
    if constexpr (W == 1) {
        r[0] = __ldg(p);
    } else if constexpr (W * sizeof(T) == 16) {
        typename V16<T>::type v = __ldg(reinterpret_cast<const typename V16<T>::type*>(p));
        const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
        for (int w = 0; w < W; ++w) r[w] = e[w];
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) r[w] = __ldg(p + w);
    }
}

template <typename T, int W>
__device__ __forceinline__ void store_vec(T* p, const T (&r)[W])
{
    if constexpr (W * sizeof(T) == 16) {
        typename V16<T>::type v;
        T* e = reinterpret_cast<T*>(&v);
#pragma unroll
        for (int w = 0; w < W; ++w) e[w] = r[w];
        *reinterpret_cast<typename V16<T>::type*>(p) = v;
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) p[w] = r[w];
    }
}

__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }

// ---------------------------------------------------------------------------------------------
// simt_gemm: the slice-GEMM (tiles in gemm_f32.cuh and gemm_f64.cuh).
//   AK   : A is K-major (inner == 1, fibres contiguous); otherwise rows (i) are contiguous.
//   VEC  : 16-byte copies of A (alignment and divisibility checked by the host).
//   BCM  : B column-major.
// Column tiles of a row tile are next to one another in the grid, so that they share A's rows in
// L2. With gridDim.z > 1 the l loop is split: part z covers l in [z * lper, min(n_q, (z + 1) *
// lper)) and writes its partial tile into ws + z * (outer * m * inner), a buffer with C's own
// layout; split_reduce_kernel then adds the parts in a fixed order, so the result does not depend
// on scheduling.
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void split_range(View3& v, int64_t lper, T* ws, int64_t& l0, int64_t& l1)
{
    l0 = 0;
    l1 = v.nq;
    if (gridDim.z > 1) {
        l0 = (int64_t)blockIdx.z * lper;
        l1 = l0 + lper < v.nq ? l0 + lper : v.nq;
        v.c = ws + (size_t)blockIdx.z * (size_t)(v.outer * v.m * v.inner);
    }
}

// Blocks per SM of the FP32 builds: 16 warps of at most 128 registers, or 20 of 100 where the accumulators
// are small (and not folded); for contiguous fibres, whose rows of A are padded further, as many as
// their shared memory lets in. The launch bounds and the walking form's grid both follow these.
constexpr int ffma_blocks(int TX, int TM, int TN, bool AK)
{
    return TX == 8 ? 2 : TM == 8 ? (AK ? 3 : 4) : AK || TN <= 4 ? 4 : 5;
}
// Shared memory of an SM, of which each block takes 1 KB besides its own.
constexpr size_t kSmSharedBytes = 228 * 1024;
constexpr bool blocks_fit(int blocks, size_t smem) { return blocks * (smem + 1024) <= kSmSharedBytes; }

template <int TX, int TM, int TN, int ST, bool AK, bool VEC, bool BCM, bool HALF>
__global__ void __launch_bounds__(32 * TX, ffma_blocks(TX, TM, TN, AK)) ffma_gemm_kernel(View3 v, ColumnGrid gr, int64_t tiles,
                                                                               int64_t lper, float* ws)
{
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    int64_t l0, l1;
    split_range(v, lper, ws, l0, l1);
    f32::tiles<TX, TM, TN, ST, AK, VEC, BCM, true, HALF>(v, blockIdx.x, gridDim.x, tiles, gr,
                                                   *reinterpret_cast<f32::Smem<TX, TM, TN, ST, AK>*>(gemm_smem), l0, l1);
}

// Blocks per SM of the FP64 builds (tiles of 64 rows of fibres: four by their shared memory; with folded
// sums by their registers).
constexpr int dmma_blocks(int BM, bool AK, int FOLD) { return BM == 128 ? 2 : AK || FOLD ? 4 : 5; }

template <int BM, int NF, int ST, bool AK, bool VEC, bool BCM, int FOLD>
__global__ void __launch_bounds__(2 * BM, dmma_blocks(BM, AK, FOLD)) dmma_gemm_kernel(View3 v, ColumnGrid gr, int64_t tiles,
                                                                             int64_t lper, double* ws)
{
    extern __shared__ __align__(16) unsigned char gemm_smem[];
    int64_t l0, l1;
    split_range(v, lper, ws, l0, l1);
    f64::tiles<BM, NF, ST, AK, VEC, BCM, true, FOLD>(v, blockIdx.x, gridDim.x, tiles, gr,
                                               *reinterpret_cast<f64::Smem<BM, NF, ST, AK, BCM>*>(gemm_smem), l0, l1);
}

// ---------------------------------------------------------------------------------------------
// colvec: small m (<= MB), strided fibres (inner >= 2). Each lane owns W consecutive rows (i of
// one slice; 16-byte loads when W = 16/sizeof(T)). The block's 8 warps are split into 8/LS row
// chunks of LS warps each; the LS warps of a chunk split the l loop (warp w takes l = w, w+LS,
// ...) and reduce through shared memory at the end. LS = 1 gives 8*32*W rows per block and no
// reduction (problems with many rows); LS = 8 gives 32*W rows per block and 8 independent load
// streams per row chunk (problems with few rows). B is staged in shared memory as [l][MB].
// ---------------------------------------------------------------------------------------------
constexpr int kColWarps = 8;
constexpr int64_t kBvecSmallMaxRows = 65536;   // small m: the l-split kernels' row tiles up to this many rows
constexpr int64_t kColSplitWarps = 148 * 32;   // fewer warps of rows than this: l split over eight warps

template <typename T, int MB>
struct ColvecSmem {
    static constexpr int MBP = MB < 4 ? 4 : MB;
    static constexpr int LB = (32768 / (MBP * (int)sizeof(T))) < 512 ? 32768 / (MBP * (int)sizeof(T)) : 512;  // l per staged chunk of B
    __align__(16) T bs[LB][MBP];
    __align__(16) T red[kColWarps][32 * (16 / sizeof(T))];
};

template <typename T, int MB, int W, int LS>
__device__ __forceinline__ void colvec_tile(const View3& v, int64_t row0, ColvecSmem<T, MB>& sm)
{
    constexpr int LB = ColvecSmem<T, MB>::LB;
    constexpr int MBP = MB < 4 ? 4 : MB;
    const T* __restrict__ A = static_cast<const T*>(v.a);
    const T* __restrict__ B = static_cast<const T*>(v.b);
    T* __restrict__ Cp = static_cast<T*>(v.c);
    const int64_t inner = v.inner, nq = v.nq, m = v.m;
    const int64_t M = v.outer * inner;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int chunk = warp / LS, part = warp % LS;
    const int64_t row = row0 + ((int64_t)chunk * 32 + lane) * W;
    const bool valid = row < M;
    const int64_t k = valid ? row / inner : 0;
    const int64_t i = valid ? row - k * inner : 0;
    const T* ap = A + k * inner * nq + i;

    T acc[MB][W];
#pragma unroll
    for (int j = 0; j < MB; ++j)
#pragma unroll
        for (int w = 0; w < W; ++w) acc[j][w] = T(0);

    for (int64_t l0 = 0; l0 < nq; l0 += LB) {
        const int lc = (int)((nq - l0) < LB ? (nq - l0) : LB);
        __syncthreads();
        for (int e = threadIdx.x; e < lc * MBP; e += blockDim.x) {
            const int l = e / MBP, j = e % MBP;
            const int64_t gl = l0 + l;
            sm.bs[l][j] = (j < m) ? (v.b_cm ? B[j + gl * m] : B[j * nq + gl]) : T(0);
        }
        __syncthreads();
        if (valid) {
#pragma unroll 4
            for (int l = part; l < lc; l += LS) {
                T a[W];
                load_vec<T, W>(a, ap + (l0 + l) * inner);
                T bj[MBP];
                if constexpr (MBP * sizeof(T) % 16 == 0) {
#pragma unroll
                    for (int c = 0; c < MBP * (int)sizeof(T) / 16; ++c) {
                        typename V16<T>::type t = *reinterpret_cast<const typename V16<T>::type*>(&sm.bs[l][c * (16 / sizeof(T))]);
#pragma unroll
                        for (int e = 0; e < (int)(16 / sizeof(T)); ++e) bj[c * (16 / sizeof(T)) + e] = reinterpret_cast<const T*>(&t)[e];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < MBP; ++j) bj[j] = sm.bs[l][j];
                }
#pragma unroll
                for (int j = 0; j < MB; ++j)
#pragma unroll
                    for (int w = 0; w < W; ++w) acc[j][w] = fma_t(a[w], bj[j], acc[j][w]);
            }
        }
    }
    T* cp = Cp + k * inner * m + i;
    if constexpr (LS == 1) {
        if (valid) {
#pragma unroll
            for (int j = 0; j < MB; ++j)
                if (j < m) store_vec<T, W>(cp + j * inner, acc[j]);
        }
    } else {
        // Reduce the LS warps' partial sums, one output column at a time.
#pragma unroll
        for (int j = 0; j < MB; ++j) {
            if (j >= m) break;
            __syncthreads();
#pragma unroll
            for (int w = 0; w < W; ++w) sm.red[warp][lane * W + w] = acc[j][w];
            __syncthreads();
            if (part == 0 && valid) {
                T r[W];
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    T t = T(0);
#pragma unroll
                    for (int q = 0; q < LS; ++q) t += sm.red[chunk * LS + q][lane * W + w];
                    r[w] = t;
                }
                store_vec<T, W>(cp + j * inner, r);
            }
        }
    }
}

template <typename T, int MB, int W, int LS>
__global__ void __launch_bounds__(256) colvec_kernel(View3 v)
{
    __shared__ ColvecSmem<T, MB> sm;
    colvec_tile<T, MB, W, LS>(v, (int64_t)blockIdx.x * (kColWarps / LS) * 32 * W, sm);
}

// colvec_async: the column kernel for rows without 16-byte alignment (one row per lane). Each
// thread streams its own row's elements A[k][l][i] into a ring of shared memory with 4- or 8-byte
// asynchronous copies (cp.async, any 4-byte alignment), kColAsyncStages - 1 stages of LC l
// (8 float, 4 double) ahead of the one it multiplies, so that many loads are in flight without
// holding them in registers. A thread reads back only what it copied itself: the ring needs no block barrier,
// only the thread's own wait on its copy groups. B is staged per chunk of LB l as in colvec.
constexpr int kColAsyncStages = 4;

template <typename T, int MB>
struct ColvecAsyncSmem {
    static constexpr int MBP = MB < 4 ? 4 : MB;
    static constexpr int LC = sizeof(T) == 8 ? 4 : 8;                      // l per stage
    static constexpr int LB = sizeof(T) == 8 ? 64 : 128;                   // l of B per chunk
    __align__(16) T a[kColAsyncStages][LC][256];
    __align__(16) T bs[LB][MBP];
    __align__(16) T red[kColWarps][32];
};

__device__ __forceinline__ void cp_async_elem(void* smem_dst, const void* src, int bytes, int src_bytes)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
    if (bytes == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T, int MB, int LS>
__device__ __forceinline__ void colvec_async_tile(const View3& v, int64_t row0, ColvecAsyncSmem<T, MB>& sm)
{
    using SM = ColvecAsyncSmem<T, MB>;
    constexpr int LB = SM::LB, LC = SM::LC, MBP = SM::MBP, ST = kColAsyncStages;
    const T* __restrict__ A = static_cast<const T*>(v.a);
    const T* __restrict__ B = static_cast<const T*>(v.b);
    T* __restrict__ Cp = static_cast<T*>(v.c);
    const int64_t inner = v.inner, nq = v.nq, m = v.m;
    const int64_t M = v.outer * inner;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chunk = warp / LS, part = warp % LS;
    const int64_t row = row0 + (int64_t)chunk * 32 + lane;
    const bool valid = row < M;
    const int64_t k = valid ? row / inner : 0;
    const int64_t i = valid ? row - k * inner : 0;
    const T* ap = A + k * inner * nq + i;

    T acc[MB];
#pragma unroll
    for (int j = 0; j < MB; ++j) acc[j] = T(0);

    for (int64_t l0 = 0; l0 < nq; l0 += LB) {
        const int lc = (int)((nq - l0) < LB ? (nq - l0) : LB);
        __syncthreads();
        for (int e = tid; e < lc * MBP; e += blockDim.x) {
            const int l = e / MBP, j = e % MBP;
            const int64_t gl = l0 + l;
            sm.bs[l][j] = (j < m) ? (v.b_cm ? B[j + gl * m] : B[j * nq + gl]) : T(0);
        }
        __syncthreads();
        // this thread's l in the chunk: part, part + LS, ...; n of them, in stages of LC
        const int n = lc > part ? (lc - part + LS - 1) / LS : 0;
        const int nst = (n + LC - 1) / LC;
        const T* base = ap + l0 * inner;
        auto issue = [&](int st) {
            T* dst = &sm.a[st % ST][0][tid];
#pragma unroll
            for (int c = 0; c < LC; ++c) {
                const int idx = st * LC + c;
                const bool ok = valid && idx < n;
                cp_async_elem(dst + c * 256, ok ? base + (int64_t)(part + idx * LS) * inner : A, (int)sizeof(T),
                              ok ? (int)sizeof(T) : 0);
            }
        };
        // one commit group per stage (empty ones too), so that wait_group counts stages
#pragma unroll
        for (int st = 0; st < ST - 1; ++st) {
            if (st < nst) issue(st);
            cp_async_commit();
        }
        for (int st = 0; st < nst; ++st) {
            // refill the slot the previous stage used, then wait for this stage's copies
            if (st + ST - 1 < nst) issue(st + ST - 1);
            cp_async_commit();
            cp_async_wait<ST - 1>();
#pragma unroll
            for (int c = 0; c < LC; ++c) {
                const int idx = st * LC + c;
                if (idx >= n) break;
                const T a = sm.a[st % ST][c][tid];
                const int l = part + idx * LS;
                T bj[MBP];
                if constexpr (MBP * sizeof(T) % 16 == 0) {
#pragma unroll
                    for (int q = 0; q < MBP * (int)sizeof(T) / 16; ++q) {
                        typename V16<T>::type t = *reinterpret_cast<const typename V16<T>::type*>(&sm.bs[l][q * (16 / sizeof(T))]);
#pragma unroll
                        for (int e = 0; e < (int)(16 / sizeof(T)); ++e) bj[q * (16 / sizeof(T)) + e] = reinterpret_cast<const T*>(&t)[e];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < MBP; ++j) bj[j] = sm.bs[l][j];
                }
#pragma unroll
                for (int j = 0; j < MB; ++j) acc[j] = fma_t(a, bj[j], acc[j]);
            }
        }
        cp_async_wait<0>();   // no copy into the ring is pending when the next chunk restarts it
    }
    T* cp = Cp + k * inner * m + i;
    if constexpr (LS == 1) {
        if (valid) {
#pragma unroll
            for (int j = 0; j < MB; ++j)
                if (j < m) cp[j * inner] = acc[j];
        }
    } else {
        // Reduce the LS warps' partial sums, one output column at a time.
#pragma unroll
        for (int j = 0; j < MB; ++j) {
            if (j >= m) break;
            __syncthreads();
            sm.red[warp][lane] = acc[j];
            __syncthreads();
            if (part == 0 && valid) {
                T t = T(0);
#pragma unroll
                for (int q = 0; q < LS; ++q) t += sm.red[chunk * LS + q][lane];
                cp[j * inner] = t;
            }
        }
    }
}

template <typename T, int MB, int LS>
__global__ void __launch_bounds__(256) colvec_async_kernel(View3 v)
{
    __shared__ ColvecAsyncSmem<T, MB> sm;
    colvec_async_tile<T, MB, LS>(v, (int64_t)blockIdx.x * (kColWarps / LS) * 32, sm);
}

// few_columns.cuh: rows of i off 16-byte boundaries, m <= 8, long l ranges.
template <int TN, bool BCM, bool CHAINS>
__global__ void __launch_bounds__(few::NT, 3) few_columns_kernel(View3 v, int chain)
{
    extern __shared__ __align__(16) unsigned char few_smem[];
    few::tile<TN, BCM, CHAINS>(v, blockIdx.x, chain, *reinterpret_cast<few::Smem<TN>*>(few_smem));
}

// ---------------------------------------------------------------------------------------------
// rowdot: small m (<= MB), contiguous fibres (inner == 1): C[k][j] = sum_l A[k][l] B(j,l).
// Each warp owns 32 rows; the block walks l in chunks of LC = 128/sizeof(T): every warp copies
// its 32 x LC tile of A into padded shared memory with coalesced 16-byte loads, the block stages
// B[l][MB] for the chunk, then each lane accumulates its own row from shared memory.
// ---------------------------------------------------------------------------------------------
template <typename T, int MB>
struct RowdotSmem {
    static constexpr int LC = 128 / sizeof(T);          // l per chunk (one 128-byte line per row)
    T a[8][32][LC + 1];                                  // per warp, padded rows
    __align__(16) T bs[LC][MB < 4 ? 4 : MB];
};

template <typename T, int MB, bool VEC>
__device__ __forceinline__ void rowdot_tile(const View3& v, int64_t row0, RowdotSmem<T, MB>& sm)
{
    constexpr int LC = RowdotSmem<T, MB>::LC;
    constexpr int MBP = MB < 4 ? 4 : MB;
    constexpr int RV = 16 / sizeof(T);
    const T* __restrict__ A = static_cast<const T*>(v.a);
    const T* __restrict__ B = static_cast<const T*>(v.b);
    T* __restrict__ Cp = static_cast<T*>(v.c);
    const int64_t nq = v.nq, m = v.m, rows = v.outer;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t wrow0 = row0 + warp * 32;
    const int64_t row = wrow0 + lane;
    T acc[MB];
#pragma unroll
    for (int j = 0; j < MB; ++j) acc[j] = T(0);

    for (int64_t l0 = 0; l0 < nq; l0 += LC) {
        const int lc = (int)((nq - l0) < LC ? (nq - l0) : LC);
        __syncthreads();
        // B chunk
        for (int e = threadIdx.x; e < LC * MBP; e += blockDim.x) {
            const int l = e / MBP, j = e % MBP;
            const int64_t gl = l0 + l;
            sm.bs[l][j] = (j < m && l < lc) ? (v.b_cm ? B[j + gl * m] : B[j * nq + gl]) : T(0);
        }
        // this warp's A tile: rows wrow0 .. +31, columns l0 .. l0+LC-1
        if (VEC) {
            // (LC / RV) lanes per row, 32 / (LC / RV) rows per step
            constexpr int LPR = LC / RV, RPS = 32 / LPR;
            const int r_in = lane / LPR, c = (lane % LPR) * RV;
#pragma unroll
            for (int r = r_in; r < 32; r += RPS) {
                const int64_t gr = wrow0 + r;
                T x[RV];
                if (gr < rows && c < lc) load_vec<T, RV>(x, A + gr * nq + l0 + c);
                else {
#pragma unroll
                    for (int e = 0; e < RV; ++e) x[e] = T(0);
                }
#pragma unroll
                for (int e = 0; e < RV; ++e) sm.a[warp][r][c + e] = x[e];
            }
        } else {
            // lane c copies column c of the warp's rows: the loads of RB rows go out before their
            // stores, so that many are in flight
            constexpr int RB = 16;
            const int c = lane;
#pragma unroll 1
            for (int rb = 0; rb < 32; rb += RB) {
                T x[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const int64_t gr = wrow0 + rb + r;
                    x[r] = (c < LC && c < lc && gr < rows) ? __ldg(A + gr * nq + l0 + c) : T(0);
                }
                if (c < LC) {
#pragma unroll
                    for (int r = 0; r < RB; ++r) sm.a[warp][rb + r][c] = x[r];
                }
            }
        }
        __syncthreads();
#pragma unroll 8
        for (int l = 0; l < lc; ++l) {
            const T a = sm.a[warp][lane][l];
            T bj[MBP];
            if constexpr (MBP * sizeof(T) % 16 == 0) {
#pragma unroll
                for (int cc = 0; cc < MBP * (int)sizeof(T) / 16; ++cc) {
                    typename V16<T>::type t = *reinterpret_cast<const typename V16<T>::type*>(&sm.bs[l][cc * RV]);
#pragma unroll
                    for (int e = 0; e < RV; ++e) bj[cc * RV + e] = reinterpret_cast<const T*>(&t)[e];
                }
            } else {
#pragma unroll
                for (int j = 0; j < MBP; ++j) bj[j] = sm.bs[l][j];
            }
#pragma unroll
            for (int j = 0; j < MB; ++j) acc[j] = fma_t(a, bj[j], acc[j]);
        }
    }
    if (row < rows) {
#pragma unroll
        for (int j = 0; j < MB; ++j)
            if (j < m) Cp[row * m + j] = acc[j];
    }
}

template <typename T, int MB, bool VEC>
__global__ void __launch_bounds__(256) rowdot_kernel(View3 v)
{
    __shared__ RowdotSmem<T, MB> sm;
    rowdot_tile<T, MB, VEC>(v, (int64_t)blockIdx.x * 256, sm);
}

// ---------------------------------------------------------------------------------------------
// rowwarp: small m (<= MB <= 8), float fibres whose ends are not on 16-byte boundaries (inner == 1).
// A warp takes R rows at a time, lanes along l: its loads are 128 contiguous bytes whatever the
// alignment, and a value of B from shared memory serves R rows. The R * MB sums of 32 lanes are
// reduced by halving: a lane ends with one output (or a group of lanes with the same one), so that a
// warp's outputs leave in one store. B's n_q <= kRowWarpNq columns are staged once per block.
// The tile kernel above copied such rows through shared memory an element at a time: fibres of 1023,
// m = 1 130 -> 46 us (3.5 TB/s), m = 8 188 -> 81 us; of 99, m = 2 56 -> 40 us. At m = 8 the reads of B
// bind it (a warp's 1 KB of B per 512 bytes of A).
// ---------------------------------------------------------------------------------------------
constexpr int kRowWarpNq = 1024;

template <int MB>
__global__ void __launch_bounds__(256) rowwarp_kernel(View3 v)
{
    constexpr int R = MB == 8 ? 4 : 8, N = R * MB;
    extern __shared__ __align__(16) float rw_smem[];   // [j][l], l padded with zeros to a multiple of 32
    const float* __restrict__ A = static_cast<const float*>(v.a);
    const float* __restrict__ B = static_cast<const float*>(v.b);
    float* __restrict__ C = static_cast<float*>(v.c);
    const int nq = (int)v.nq, m = (int)v.m, np = (nq + 31) / 32 * 32;
    for (int e = threadIdx.x; e < MB * np; e += 256) {
        const int j = e / np, l = e - j * np;
        rw_smem[e] = j < m && l < nq ? (v.b_cm ? B[j + (int64_t)l * m] : B[(int64_t)j * nq + l]) : 0.0f;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t rows = v.outer, warps = (int64_t)gridDim.x * 8;
    for (int64_t g = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); g * R < rows; g += warps) {
        const int64_t row0 = g * R;
        const int have = (int)(rows - row0 < R ? rows - row0 : R);
        const float* p = A + row0 * nq + lane;
        float acc[N];
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = 0.0f;
#pragma unroll 2
        for (int l0 = 0; l0 < np; l0 += 32) {
            const bool ok = l0 + lane < nq;
            float a[R], b[MB];
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = ok && r < have ? __ldg(p + (int64_t)r * nq + l0) : 0.0f;
#pragma unroll
            for (int j = 0; j < MB; ++j) b[j] = rw_smem[j * np + l0 + lane];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int j = 0; j < MB; ++j) acc[r * MB + j] = __fmaf_rn(a[r], b[j], acc[r * MB + j]);
        }
        // output i ends in lanes i * 32 / N ..
        int n = N;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            if (n > 1) {
                n /= 2;
                const bool up = lane & s;
#pragma unroll
                for (int i = 0; i < N / 2; ++i) {
                    if (i < n) {
                        const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
                        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
                    }
                }
            } else {
                acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], s);
            }
        }
        constexpr int G = 32 / N;   // lanes that hold the same output
        const int i = lane / G, r = i / MB, j = i % MB;
        if (lane % G == 0 && r < have && j < m) C[(row0 + r) * m + j] = acc[0];
    }
}

// ---------------------------------------------------------------------------------------------
// rowflat: small m, contiguous fibres of at most kFlatMaxNq elements (inner == 1, short rows).
// A warp's wr consecutive rows are wr * nq contiguous elements: the warp copies them with
// coalesced loads into shared memory with rows padded to nq + 1 (conflict-free row reads), then
// each lane computes every 32nd row. B sits in shared memory as bs[l][j]. With STAGE, the m
// outputs of 32 consecutive rows (32 * m contiguous elements of C) are staged in shared memory
// (rows padded to an odd stride) and written with coalesced stores, 32 consecutive elements per
// instruction; without it each lane stores its own row (a stride of m elements between lanes),
// which measured faster where a row's outputs are short or the fibres long.
// ---------------------------------------------------------------------------------------------
constexpr int kFlatMaxNq = 16;

template <typename T, int MB, bool STAGE>
__global__ void __launch_bounds__(256) rowflat_kernel(View3 v, int wr)
{
    constexpr int MBP = MB < 4 ? 4 : MB;
    extern __shared__ __align__(16) unsigned char flat_raw[];
    T* smf = reinterpret_cast<T*>(flat_raw);
    const int nq = (int)v.nq, stride = nq + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* tile = smf + (size_t)warp * wr * stride;
    T* bs = smf + (size_t)8 * wr * stride;
    const T* __restrict__ B = static_cast<const T*>(v.b);
    for (int e = threadIdx.x; e < nq * MBP; e += blockDim.x) {
        const int l = e / MBP, j = e - l * MBP;
        bs[e] = j < v.m ? (v.b_cm ? B[j + (int64_t)l * v.m] : B[(int64_t)j * nq + l]) : T(0);
    }
    __syncthreads();
    const int64_t wrow0 = ((int64_t)blockIdx.x * 8 + warp) * wr;
    if (wrow0 >= v.outer) return;
    const int nrow = (int)((v.outer - wrow0) < wr ? (v.outer - wrow0) : wr);
    const T* __restrict__ A = static_cast<const T*>(v.a) + wrow0 * nq;
    const int cnt = nrow * nq;
    // e / nq == umulhi(e, ceil(2^32 / nq)) for these e (nq > 1; 2^32 itself does not fit)
    const uint32_t inv = nq > 1 ? (uint32_t)((0x100000000ull + nq - 1) / nq) : 0u;
#pragma unroll 16
    for (int e = lane; e < cnt; e += 32) {
        const int r = nq > 1 ? (int)__umulhi((uint32_t)e, inv) : e;
        tile[r * stride + (e - r * nq)] = __ldg(A + e);
    }
    __syncwarp();
    T* __restrict__ Cp = static_cast<T*>(v.c);
    const int m = (int)v.m;
    if constexpr (!STAGE) {
        for (int r = lane; r < nrow; r += 32) {
            T acc[MB];
#pragma unroll
            for (int j = 0; j < MB; ++j) acc[j] = T(0);
            const T* row = tile + r * stride;
            for (int l = 0; l < nq; ++l) {
                const T a = row[l];
#pragma unroll
                for (int j = 0; j < MB; ++j) acc[j] = fma_t(a, bs[l * MBP + j], acc[j]);
            }
            T* cp = Cp + (wrow0 + r) * (int64_t)m;
#pragma unroll
            for (int j = 0; j < MB; ++j)
                if (j < m) cp[j] = acc[j];
        }
        return;
    }
    // staged: this warp's 32 x (m | 1) outputs after B (odd row stride, conflict-free writes)
    const int ms = m | 1;
    T* ostage = bs + (size_t)nq * MBP + (size_t)warp * 32 * ms;
    // e / m == umulhi(e, ceil(2^32 / m)) for e < 32 * m (m > 1)
    const uint32_t minv = m > 1 ? (uint32_t)((0x100000000ull + m - 1) / m) : 0u;
    for (int r0 = 0; r0 < nrow; r0 += 32) {
        const int r = r0 + lane;
        if (r < nrow) {
            T acc[MB];
#pragma unroll
            for (int j = 0; j < MB; ++j) acc[j] = T(0);
            const T* row = tile + r * stride;
            for (int l = 0; l < nq; ++l) {
                const T a = row[l];
#pragma unroll
                for (int j = 0; j < MB; ++j) acc[j] = fma_t(a, bs[l * MBP + j], acc[j]);
            }
#pragma unroll
            for (int j = 0; j < MB; ++j)
                if (j < m) ostage[lane * ms + j] = acc[j];
        }
        __syncwarp();
        // rows r0 .. r0 + nr - 1: nr * m contiguous outputs from C[(wrow0 + r0) * m]
        const int nr = (nrow - r0) < 32 ? (nrow - r0) : 32;
        T* cp = Cp + (wrow0 + r0) * (int64_t)m;
        for (int e = lane; e < nr * m; e += 32) {
            const int rr = m > 1 ? (int)__umulhi((uint32_t)e, minv) : e;
            cp[e] = ostage[rr * ms + (e - rr * m)];
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------------
// rowspan: small m, contiguous fibres of NQ in {1, 2, 4, 8, 16} elements (at most a span), A
// 16-byte aligned. Thread t reads the 64-byte span (16 floats / 8 doubles) holding the R = span /
// NQ whole fibres t*R .. t*R + R-1 with 128-bit loads: consecutive threads read consecutive
// spans, so a warp's loads are fully coalesced and nothing is staged. Its R*m outputs are
// contiguous in C. B sits in shared memory (broadcast reads). Used where a thread's outputs take
// at most 64 bytes (measured: more outputs per thread scatter the stores too widely).
// ---------------------------------------------------------------------------------------------
template <typename T, int MB, int NQ>
__global__ void __launch_bounds__(256) rowspan_kernel(View3 v)
{
    constexpr int E = 64 / (int)sizeof(T), R = E / NQ, VW = 16 / (int)sizeof(T), NV = E / VW;
    static_assert(NQ <= E, "a fibre fits a span");
    __shared__ T bs[NQ * MB];
    const T* __restrict__ B = static_cast<const T*>(v.b);
    for (int e = threadIdx.x; e < NQ * MB; e += blockDim.x) {
        const int l = e / MB, j = e - l * MB;
        bs[e] = j < v.m ? (v.b_cm ? B[j + (int64_t)l * v.m] : B[(int64_t)j * NQ + l]) : T(0);
    }
    __syncthreads();
    const T* __restrict__ A = static_cast<const T*>(v.a);
    T* __restrict__ Cp = static_cast<T*>(v.c);
    const int64_t rows = v.outer, spans = (rows + R - 1) / R;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < spans; t += stride) {
        const int64_t r0 = t * R;
        T a[E];
        if (r0 + R <= rows) {
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                T x[VW];
                load_vec<T, VW>(x, A + r0 * NQ + q * VW);
#pragma unroll
                for (int w = 0; w < VW; ++w) a[q * VW + w] = x[w];
            }
        } else {
#pragma unroll
            for (int e = 0; e < E; ++e) a[e] = (r0 + e / NQ < rows) ? __ldg(A + r0 * NQ + e) : T(0);
        }
        T* cp = Cp + r0 * v.m;
        // R*m contiguous outputs: with m == MB, a 16-byte aligned C and R*MB a multiple of VW,
        // written VW at a time (a vector covers MB / VW of a row, or VW / MB rows)
        const bool vec = r0 + R <= rows && v.m == MB && (R * MB) % VW == 0 &&
                         (reinterpret_cast<uintptr_t>(cp) & 15u) == 0;
        if (vec) {
#pragma unroll
            for (int q = 0; q < R * MB / VW; ++q) {
                T x[VW];
#pragma unroll
                for (int w = 0; w < VW; ++w) {
                    const int o = q * VW + w, r = o / MB, j = o - r * MB;
                    T acc = T(0);
#pragma unroll
                    for (int l = 0; l < NQ; ++l) acc = fma_t(a[r * NQ + l], bs[l * MB + j], acc);
                    x[w] = acc;
                }
                store_vec<T, VW>(cp + q * VW, x);
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (r0 + r >= rows) break;
#pragma unroll
                for (int j = 0; j < MB; ++j) {
                    if (j >= v.m) break;
                    T acc = T(0);
#pragma unroll
                    for (int l = 0; l < NQ; ++l) acc = fma_t(a[r * NQ + l], bs[l * MB + j], acc);
                    cp[(int64_t)r * v.m + j] = acc;
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// strided: one thread per C element, strides taken from the caller.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) strided_kernel(StridedProblem sp)
{
    const T* __restrict__ A = static_cast<const T*>(sp.a);
    const T* __restrict__ B = static_cast<const T*>(sp.b);
    T* __restrict__ Cp = static_cast<T*>(sp.c);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < sp.total; e += stride) {
        int64_t rem = e, aoff = 0, coff = 0, j = 0;
        for (int r = 0; r < sp.p; ++r) {
            const int mode = sp.order[r];
            const int64_t ext = sp.nc[mode];
            const int64_t idx = rem % ext;
            rem /= ext;
            coff += idx * sp.wc[mode];
            if (mode == sp.q) j = idx;
            else aoff += idx * sp.wa[mode];
        }
        const int64_t wq = sp.wa[sp.q];
        T acc = T(0);
        for (int64_t l = 0; l < sp.nq; ++l) {
            const T bv = sp.b_cm ? B[j + l * sp.m] : B[j * sp.nq + l];
            acc = fma_t(A[aoff + l * wq], bv, acc);
        }
        Cp[coff] = acc;
    }
}

// ---------------------------------------------------------------------------------------------
// grouped: many independent TTMs in one persistent launch. Blocks pull work items from a device
// counter; an item is one slice-GEMM tile of a problem (m > 16) or a block of 256 rows of a
// small-m problem. Problems are ordered largest first by the host, so the tail is short.
// ---------------------------------------------------------------------------------------------
template <typename T>
union SmallSmem {
    ColvecAsyncSmem<T, 16> cola;
    RowdotSmem<T, 16> row;
};

// One small-m work item: 256 rows of contiguous fibres, or of one strided fibre per lane.
template <typename T, int MB>
__device__ __forceinline__ void grouped_small(const View3& v, int flags, int64_t local, SmallSmem<T>& sm)
{
    auto& row = reinterpret_cast<RowdotSmem<T, MB>&>(sm.row);
    if (flags & 1) {
        if (flags & 2) rowdot_tile<T, MB, true>(v, local * 256, row);
        else rowdot_tile<T, MB, false>(v, local * 256, row);
    } else {
        colvec_async_tile<T, MB, 1>(v, local * kColWarps * 32, reinterpret_cast<ColvecAsyncSmem<T, MB>&>(sm.cola));
    }
}

constexpr int kGroupNF = 8, kGroupST = 3;   // the FP64 tile of the grouped launch
template <typename T>
constexpr size_t grouped_smem_bytes()
{
    if (sizeof(T) == 4)
        return std::max(sizeof(f32::Smem<8, kGemmRows / 32, kGroupNF, kGroupST, true>),
                        sizeof(f32::Smem<8, kGemmRows / 32, kGroupNF, kGroupST, false>));
    const size_t rows = sizeof(f64::Smem<kGemmRows, kGroupNF, kGroupST, true, false>),
                 cols = sizeof(f64::Smem<kGemmRows, kGroupNF, kGroupST, false, true>);
    return std::max(rows, cols);   // the largest of the four forms: one pitch of A with one of B
}

#define TLIBTTM_TILES                                                                                \
    if (ak) {                                                                                        \
        if (vec) { if (g.b_cm) TLIBTTM_TILE(true, true, true); else TLIBTTM_TILE(true, true, false); } \
        else     { if (g.b_cm) TLIBTTM_TILE(true, false, true); else TLIBTTM_TILE(true, false, false); } \
    } else {                                                                                         \
        if (vec) { if (g.b_cm) TLIBTTM_TILE(false, true, true); else TLIBTTM_TILE(false, true, false); } \
        else     { if (g.b_cm) TLIBTTM_TILE(false, false, true); else TLIBTTM_TILE(false, false, false); } \
    }

// Two CTAs per SM (at most 128 registers; the FP64 build spills some 300 bytes a thread): measured faster
// on the batched workload than one CTA of 255 registers.
template <typename T>
__global__ void __launch_bounds__(256, 2) grouped_kernel(const GroupDesc* __restrict__ desc, int count, int64_t total,
                                                      unsigned long long* queue)
{
    extern __shared__ __align__(16) unsigned char grouped_smem[];
    __shared__ int64_t item_s;
    for (;;) {
        if (threadIdx.x == 0) item_s = (int64_t)atomicAdd(queue, 1ull);
        __syncthreads();
        const int64_t item = item_s;
        if (item >= total) break;
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (desc[mid].first <= item) lo = mid;
            else hi = mid - 1;
        }
        const GroupDesc g = desc[lo];
        const int64_t local = item - g.first;
        View3 v;
        v.a = g.a;
        v.b = g.b;
        v.c = g.c;
        v.outer = g.outer;
        v.nq = g.nq;
        v.inner = g.inner;
        v.m = g.m;
        v.b_cm = g.b_cm;
        const bool ak = g.flags & 1, vec = g.flags & 2;
        const ColumnGrid gr{g.tiles_n, g.cols / 8};
        if constexpr (sizeof(T) == 8) {
#define TLIBTTM_TILE(AKv, VECv, BCMv)                                                                        \
    f64::tiles<kGemmRows, kGroupNF, kGroupST, AKv, VECv, BCMv, false, 0>(v, local, 1, local + 1, gr,                    \
                                                   *reinterpret_cast<f64::Smem<kGemmRows, kGroupNF, kGroupST, AKv, BCMv>*>(grouped_smem), \
                                                   0, v.nq)
            TLIBTTM_TILES
#undef TLIBTTM_TILE
        } else {
#define TLIBTTM_TILE(AKv, VECv, BCMv)                                                                                 \
    f32::tiles<8, kGemmRows / 32, kGroupNF, kGroupST, AKv, VECv, BCMv, false>(v, local, 1, local + 1, gr,                \
                                                                           *reinterpret_cast<f32::Smem<8, kGemmRows / 32, kGroupNF, kGroupST, AKv>*>(grouped_smem), \
                                                                           0, v.nq)
            TLIBTTM_TILES
#undef TLIBTTM_TILE
        }
        __syncthreads();
    }
}

// Grouped launch of small-m problems only: the same work items as grouped_kernel's small-m ones,
// without the slice-GEMM's registers and shared memory, so that more blocks share an SM (their
// loads in flight are what these bandwidth-bound items need). Measured against one launch per
// MB build (each launch leaves a tail) and against the MB = 16 build for every item (small m then
// computes 16 columns): one launch that picks the build per item is the fastest of the three. A
// block's items come from the queue in increasing order, so the problem search goes on from the
// previous item's.
template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 4 : 2) grouped_small_kernel(const GroupDesc* __restrict__ desc, int count,
                                                           int64_t total, unsigned long long* queue)
{
    __shared__ SmallSmem<T> sm;
    __shared__ int64_t item_s;
    int cur = 0;
    for (;;) {
        if (threadIdx.x == 0) item_s = (int64_t)atomicAdd(queue, 1ull);
        __syncthreads();
        const int64_t item = item_s;
        if (item >= total) break;
        while (cur + 1 < count && desc[cur + 1].first <= item) ++cur;
        const GroupDesc g = desc[cur];
        const int64_t local = item - g.first;
        View3 v;
        v.a = g.a;
        v.b = g.b;
        v.c = g.c;
        v.outer = g.outer;
        v.nq = g.nq;
        v.inner = g.inner;
        v.m = g.m;
        v.b_cm = g.b_cm;
        if (g.m <= 1) grouped_small<T, 1>(v, g.flags, local, sm);
        else if (g.m <= 2) grouped_small<T, 2>(v, g.flags, local, sm);
        else if (g.m <= 4) grouped_small<T, 4>(v, g.flags, local, sm);
        else if (g.m <= 8) grouped_small<T, 8>(v, g.flags, local, sm);
        else grouped_small<T, 16>(v, g.flags, local, sm);
        __syncthreads();
    }
}

int g_sms_simt = 0;

cudaError_t sms_of_device(int& sms)
{
    if (!g_sms_simt) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sms_simt, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
    }
    sms = g_sms_simt;
    return cudaSuccess;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <int TX, int TM, int TN, int ST, bool AK, bool VEC, bool BCM>
cudaError_t ffma_launch(const View3& v, cudaStream_t s, const ColumnGrid& gr, int sms, int split, int64_t lper, float* ws)
{
    constexpr int smem = (int)sizeof(f32::Smem<TX, TM, TN, ST, AK>);
    static_assert(blocks_fit(ffma_blocks(TX, TM, TN, AK), smem), "the walking form's blocks are resident at once");
    // wide tiles of contiguous fibres, short ranges: half stages (128000 fibres, m = 512: n_q = 20 125 ->
    // 99 us, n_q = 8 85 -> 69)
    auto kernel = ffma_gemm_kernel<TX, TM, TN, ST, AK, VEC, BCM, false>;
    if constexpr (AK && TX == 8)
        if (v.nq <= 4 * f32::BK) kernel = ffma_gemm_kernel<TX, TM, TN, ST, AK, VEC, BCM, true>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int64_t tiles = ceil_div(v.outer * v.inner, 32 * TM) * gr.cols;
    // as in dmma_launch (m = 64, n_q = 16, A 64 MB: 86 -> 82 us; n_q = 64: 190 us against 197); several
    // column tiles are balanced better one by one (128000 fibres of 20, m = 99: 35 us against 45)
    const bool walk = gr.cols == 1 && v.nq <= 2 * f32::BK;
    const int64_t slots = (int64_t)sms * ffma_blocks(TX, TM, TN, AK);
    const dim3 grid((unsigned)(walk ? std::min(tiles, slots) : tiles), 1, (unsigned)split);
    kernel<<<grid, 32 * TX, smem, s>>>(v, gr, tiles, lper, ws);
    return cudaGetLastError();
}

template <int TX, int TM, int TN, int ST>
cudaError_t ffma_dispatch_form(const View3& v, cudaStream_t s, const ColumnGrid& gr, int sms, int split, int64_t lper, float* ws)
{
#define TLIBTTM_FFMA(AKv, VECv) \
    (v.b_cm ? ffma_launch<TX, TM, TN, ST, AKv, VECv, true>(v, s, gr, sms, split, lper, ws) \
            : ffma_launch<TX, TM, TN, ST, AKv, VECv, false>(v, s, gr, sms, split, lper, ws))
    const bool vec = aligned16(v.a) && (v.inner == 1 ? v.nq : v.inner) % 4 == 0;
    if (v.inner == 1) return vec ? TLIBTTM_FFMA(true, true) : TLIBTTM_FFMA(true, false);
    return vec ? TLIBTTM_FFMA(false, true) : TLIBTTM_FFMA(false, false);
#undef TLIBTTM_FFMA
}

// m <= 16: whether the kernels that the slice-GEMM tile replaces add up in one chain per output, so that
// one chain of its own is no further off. They do not where the range is split here; for rows of i that
// the column kernel takes with its eight warps, for fibres that the l-split kernels take, and where the
// TMA-fed kernel may split the l range (tiles that leave SMs idle, or a last round worth splitting; its
// shape model never splits ranges below 160 l).
bool one_chain_before(const View3& v, int dtype, int split)
{
    if (split > 1) return false;
    const int64_t rows = v.outer * v.inner, rv = dtype == 0 ? 4 : 2;
    const bool tma = rows * v.nq * (16 / rv) >= kStreamMinBytes && stream_supported(v, dtype);
    if (v.inner == 1) return tma ? rows >= 148 * 512 && v.nq <= 1024 : rows > kBvecSmallMaxRows || v.nq < 1024;
    if (tma) return v.nq < 160 || (rows >= 2 * 148 * 256 * rv && v.nq <= 1024);
    const int64_t w = aligned16(v.a) && aligned16(v.c) && v.inner % rv == 0 ? rv : 1;   // rows per lane
    return rows > kColSplitWarps * 32 * w;
}

// At most 16 columns: tiles of 256 rows in one chain where that is no further off and they fill the GPU
// (four blocks per SM), else tiles of 128 rows in folded sums, whose levels fit the registers.
template <int TM, int ST>
cudaError_t ffma_dispatch_small(const View3& v, cudaStream_t s, int sms, int split, int64_t lper, float* ws)
{
    const ColumnGrid gr = split_columns(v.m, 4, 4);
    switch (gr.nf) {
    case 1: return ffma_dispatch_form<4, TM, 1, ST>(v, s, gr, sms, split, lper, ws);
    case 2: return ffma_dispatch_form<4, TM, 2, ST>(v, s, gr, sms, split, lper, ws);
    case 3: return ffma_dispatch_form<4, TM, 3, ST>(v, s, gr, sms, split, lper, ws);
    default: return ffma_dispatch_form<4, TM, 4, ST>(v, s, gr, sms, split, lper, ws);
    }
}

template <int TM, int ST>
cudaError_t ffma_dispatch_narrow(const View3& v, cudaStream_t s, int sms, int split, int64_t lper, float* ws)
{
    const ColumnGrid gr = split_columns(v.m, 8, 4);
    switch (gr.nf) {
    case 5: return ffma_dispatch_form<4, TM, 5, ST>(v, s, gr, sms, split, lper, ws);
    case 6: return ffma_dispatch_form<4, TM, 6, ST>(v, s, gr, sms, split, lper, ws);
    case 7: return ffma_dispatch_form<4, TM, 7, ST>(v, s, gr, sms, split, lper, ws);
    default: return ffma_dispatch_form<4, TM, 8, ST>(v, s, gr, sms, split, lper, ws);
    }
}

cudaError_t simt_gemm_dispatch(const View3& v, cudaStream_t s, int split = 1, int64_t lper = 0, float* ws = nullptr)
{
    int sms = 0;
    const cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    const int64_t rows = (split > 1 ? split : 1) * ceil_div(v.outer * v.inner, 256);
    if (v.m <= kSmallM)
        return rows >= 4 * sms && one_chain_before(v, 0, split) ? ffma_dispatch_small<8, 3>(v, s, sms, split, lper, ws)
                                                                : ffma_dispatch_small<4, 4>(v, s, sms, split, lper, ws);
    // Blocks of 8 x 8 outputs a thread where they fill both slots of every SM; up to 32 columns, and
    // problems with fewer tiles, in the narrow form (its shared-memory reads per multiply-add are
    // those of the wide form at half the columns: m = 24, A 160 MB 74 -> 59 us), with rows of 128
    // where 256 would leave slots empty, or be padding for a quarter of its rows or more (split ranges of
    // few rows: A (128, 2^17), m = 256 430 -> 231 us, (300, 2^17), m = 100 402 -> 316).
    const bool tall = 5 * ceil_div(v.outer * v.inner, 128) >= 8 * ceil_div(v.outer * v.inner, 256);
    if (v.m > 32 && tall && rows * ceil_div(v.m, 64) >= 2 * sms) {
        const ColumnGrid gr = split_columns(v.m, 8);
        switch (gr.nf) {
        case 5: return ffma_dispatch_form<8, 8, 5, 4>(v, s, gr, sms, split, lper, ws);
        case 6: return ffma_dispatch_form<8, 8, 6, 4>(v, s, gr, sms, split, lper, ws);
        case 7: return ffma_dispatch_form<8, 8, 7, 4>(v, s, gr, sms, split, lper, ws);
        default: return ffma_dispatch_form<8, 8, 8, 4>(v, s, gr, sms, split, lper, ws);
        }
    }
    return tall && rows * ceil_div(v.m, 32) >= 4 * sms ? ffma_dispatch_narrow<8, 3>(v, s, sms, split, lper, ws)
                                                   : ffma_dispatch_narrow<4, 4>(v, s, sms, split, lper, ws);
}

template <int BM, int NF, int ST, bool AK, bool VEC, bool BCM, int FOLD>
cudaError_t dmma_launch(const View3& v, cudaStream_t s, const ColumnGrid& gr, int sms, int split, int64_t lper, double* ws)
{
    constexpr int smem = (int)sizeof(f64::Smem<BM, NF, ST, AK, BCM>);
    static_assert(blocks_fit(dmma_blocks(BM, AK, FOLD), smem), "the walking form's blocks are resident at once");
    const auto kernel = dmma_gemm_kernel<BM, NF, ST, AK, VEC, BCM, FOLD>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int64_t tiles = ceil_div(v.outer * v.inner, BM) * gr.cols;
    // Short l ranges: a fixed set of blocks walks the tiles, so that the ring stays full across
    // them (n_q = 16, A 256 MB: m = 64 147 -> 114 us, m = 8 94 -> 67 us). Longer ones: a block per
    // tile, which the scheduler balances better (m = 64, n_q = 48: 97 us against 113).
    // So are several column tiles of fibres whose outputs leave one by one (128000 fibres of 8, m = 355 161
    // us against 205; m = 130, in pairs, 45 against 36).
    const bool walk = v.nq <= (NF <= 2 ? 8 : 2) * f64::BK && (gr.cols == 1 || !AK || v.m % 2 == 0);
    const int64_t slots = (int64_t)sms * dmma_blocks(BM, AK, FOLD);
    const dim3 grid((unsigned)(walk ? std::min(tiles, slots) : tiles), 1, (unsigned)split);
    kernel<<<grid, 2 * BM, smem, s>>>(v, gr, tiles, lper, ws);
    return cudaGetLastError();
}

template <int BM, int NF, int ST, bool AK, bool VEC>
cudaError_t dmma_dispatch_form(const View3& v, cudaStream_t s, const ColumnGrid& gr, int sms, int split, int64_t lper, double* ws,
                               int fold)
{
    if constexpr (NF <= 2) {
        if (fold == 16)
            return v.b_cm ? dmma_launch<BM, NF, ST, AK, VEC, true, 16>(v, s, gr, sms, split, lper, ws)
                          : dmma_launch<BM, NF, ST, AK, VEC, false, 16>(v, s, gr, sms, split, lper, ws);
        if constexpr (!AK)
            if (fold == 8)
                return v.b_cm ? dmma_launch<BM, NF, ST, AK, VEC, true, 8>(v, s, gr, sms, split, lper, ws)
                              : dmma_launch<BM, NF, ST, AK, VEC, false, 8>(v, s, gr, sms, split, lper, ws);
    }
    return v.b_cm ? dmma_launch<BM, NF, ST, AK, VEC, true, 0>(v, s, gr, sms, split, lper, ws)
                  : dmma_launch<BM, NF, ST, AK, VEC, false, 0>(v, s, gr, sms, split, lper, ws);
}

// BM 64: 16-byte copies of A only; 128 with one or two groups of columns: 8-byte ones only.
template <int BM, int NF, int ST>
cudaError_t dmma_dispatch_nf(const View3& v, cudaStream_t s, const ColumnGrid& gr, int sms, int split, int64_t lper, double* ws,
                             bool vec, int fold = 0)
{
    if (vec) {
        if constexpr (BM == 64 || NF > 2)
            return v.inner == 1 ? dmma_dispatch_form<BM, NF, ST, true, true>(v, s, gr, sms, split, lper, ws, fold)
                                : dmma_dispatch_form<BM, NF, ST, false, true>(v, s, gr, sms, split, lper, ws, fold);
    } else {
        if constexpr (BM == 128)
            return v.inner == 1 ? dmma_dispatch_form<BM, NF, ST, true, false>(v, s, gr, sms, split, lper, ws, fold)
                                : dmma_dispatch_form<BM, NF, ST, false, false>(v, s, gr, sms, split, lper, ws, fold);
    }
    return cudaErrorNotSupported;
}

// The length of the tile's chains (0: one chain of n_q). Chains of 8 take 5-9 % more time than those of 16
// and are as good as the column kernel's eight chains up to n_q = 160, those of 16 from there.
int dmma_chain(const View3& v, int split)
{
    if (v.m > kSmallM || one_chain_before(v, 1, split)) return 0;
    return v.inner > 1 && v.nq < 160 ? 8 : 16;
}

// Widest column tile in groups of eight: 64 columns where the tiles fill the GPU, narrower ones
// (more blocks, A's rows shared through L2) where they do not.
int dmma_width(const View3& v, int sms)
{
    const int64_t rows = ceil_div(v.outer * v.inner, 128), groups = ceil_div(v.m, 8);
    for (int nf : {8, 4})
        if (groups > nf / 2 && rows * ceil_div(groups, nf) >= sms) return nf;
    return 2;
}

cudaError_t simt_gemm_dispatch(const View3& v, cudaStream_t s, int split = 1, int64_t lper = 0, double* ws = nullptr)
{
    int sms = 0;
    const cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    const bool vec = aligned16(v.a) && (v.inner == 1 ? v.nq : v.inner) % 2 == 0;
    const ColumnGrid gr = split_columns(v.m, split > 1 ? (v.m > 16 ? 8 : 2) : dmma_width(v, sms));
    const int fold = dmma_chain(v, split);
    switch (gr.nf) {
    case 1:
        return vec ? dmma_dispatch_nf<64, 1, 4>(v, s, gr, sms, split, lper, ws, true, fold)
                   : dmma_dispatch_nf<128, 1, 4>(v, s, gr, sms, split, lper, ws, false, fold);
    case 2:
        return vec ? dmma_dispatch_nf<64, 2, 4>(v, s, gr, sms, split, lper, ws, true, fold)
                   : dmma_dispatch_nf<128, 2, 4>(v, s, gr, sms, split, lper, ws, false, fold);
    case 3: return dmma_dispatch_nf<128, 3, 4>(v, s, gr, sms, split, lper, ws, vec);
    case 4: return dmma_dispatch_nf<128, 4, 4>(v, s, gr, sms, split, lper, ws, vec);
    case 5: return dmma_dispatch_nf<128, 5, 3>(v, s, gr, sms, split, lper, ws, vec);
    case 6: return dmma_dispatch_nf<128, 6, 3>(v, s, gr, sms, split, lper, ws, vec);
    case 7: return dmma_dispatch_nf<128, 7, 3>(v, s, gr, sms, split, lper, ws, vec);
    default: return dmma_dispatch_nf<128, 8, 3>(v, s, gr, sms, split, lper, ws, vec);
    }
}

template <typename T, int W, int LS>
cudaError_t colvec_dispatch_ls(const View3& v, cudaStream_t s)
{
    const int64_t M = v.outer * v.inner;
    dim3 grid((unsigned)ceil_div(M, (kColWarps / LS) * 32 * W)), block(256);
#define TLIBTTM_COLVEC(MBv)                                                                \
    do {                                                                                   \
        if constexpr (W == 1) colvec_async_kernel<T, MBv, LS><<<grid, block, 0, s>>>(v);   \
        else colvec_kernel<T, MBv, W, LS><<<grid, block, 0, s>>>(v);                       \
    } while (0)
    if (v.m <= 1) TLIBTTM_COLVEC(1);
    else if (v.m <= 2) TLIBTTM_COLVEC(2);
    else if (v.m <= 4) TLIBTTM_COLVEC(4);
    else if (v.m <= 8) TLIBTTM_COLVEC(8);
    else TLIBTTM_COLVEC(16);
#undef TLIBTTM_COLVEC
    return cudaGetLastError();
}

template <int TN>
cudaError_t few_columns_launch(const View3& v, cudaStream_t s)
{
    constexpr int smem = (int)sizeof(few::Smem<TN>);
    // the column kernel would split l over eight warps below this many rows
    const bool chains = v.outer * v.inner <= kColSplitWarps * 32;
    const auto kernel = v.b_cm ? (chains ? few_columns_kernel<TN, true, true> : few_columns_kernel<TN, true, false>)
                               : (chains ? few_columns_kernel<TN, false, true> : few_columns_kernel<TN, false, false>);
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int chain = v.nq < 128 ? 1 : 3;
    kernel<<<(unsigned)(v.outer * ceil_div(v.inner, few::BM)), few::NT, smem, s>>>(v, chain);
    return cudaGetLastError();
}

// Measured against the column kernel on A of 160 MB, as its time over the few-column kernel's: with
// tiles full 1.2-1.6 at m = 1 from n_q = 17, 1.25-1.9 at m = 2..4 and 1.1-1.8 at m = 5..8 from n_q =
// 33 (0.75-1.0 at 17); half-full tiles (inner 129, 257) 1.2-1.3 at m = 1, 1.05-1.1 at 2..4, 0.9 at
// 5..8, and 1.04 there at 0.59 full (inner 301). Fewer tiles than this leave SMs idle, where the
// column kernel splits l.
bool few_columns_takes(const View3& v)
{
    const int64_t per_slice = ceil_div(v.inner, few::BM), room = per_slice * few::BM;
    return v.m <= 8 && v.inner % 4 != 0 && aligned16(v.a) && v.outer * per_slice >= 128 && v.nq >= (v.m == 1 ? 17 : 33) &&
           16 * v.inner >= (v.m <= 4 ? 8 : 9) * room;
}

cudaError_t few_columns_dispatch(const View3& v, cudaStream_t s)
{
    return v.m <= 1 ? few_columns_launch<1>(v, s) : v.m <= 2 ? few_columns_launch<2>(v, s)
         : v.m <= 4 ? few_columns_launch<4>(v, s) : few_columns_launch<8>(v, s);
}

// Rows per lane of the column kernel: 16 bytes of them, or one.
template <typename T>
int colvec_rows_per_lane(const View3& v)
{
    constexpr int RV = 16 / sizeof(T);
    return aligned16(v.a) && aligned16(v.c) && v.inner % RV == 0 ? RV : 1;
}

template <typename T>
cudaError_t colvec_dispatch(const View3& v, int ls, cudaStream_t s)
{
    constexpr int RV = 16 / sizeof(T);
    if (colvec_rows_per_lane<T>(v) == RV)
        return ls == 8 ? colvec_dispatch_ls<T, RV, 8>(v, s) : colvec_dispatch_ls<T, RV, 1>(v, s);
    return ls == 8 ? colvec_dispatch_ls<T, 1, 8>(v, s) : colvec_dispatch_ls<T, 1, 1>(v, s);
}

template <typename T, bool VEC>
cudaError_t rowdot_dispatch_v(const View3& v, cudaStream_t s)
{
    dim3 grid((unsigned)ceil_div(v.outer, 256)), block(256);
    if (v.m <= 1) rowdot_kernel<T, 1, VEC><<<grid, block, 0, s>>>(v);
    else if (v.m <= 2) rowdot_kernel<T, 2, VEC><<<grid, block, 0, s>>>(v);
    else if (v.m <= 4) rowdot_kernel<T, 4, VEC><<<grid, block, 0, s>>>(v);
    else if (v.m <= 8) rowdot_kernel<T, 8, VEC><<<grid, block, 0, s>>>(v);
    else rowdot_kernel<T, 16, VEC><<<grid, block, 0, s>>>(v);
    return cudaGetLastError();
}

template <typename T, int MB, bool STAGE>
cudaError_t rowflat_launch_s(const View3& v, cudaStream_t s)
{
    // rows per warp: about 4 KB of A, a multiple of 32, with the block's tiles, B and the output
    // staging (8 warps x 32 rows x (m | 1)) within 44 KB of shared memory where that allows 32 rows
    const int64_t es = (int64_t)sizeof(T), ms = STAGE ? (v.m | 1) : 0;
    const int64_t fixed = 16 * 16 * es + 8 * 32 * ms * es;
    const int64_t want = 4096 / (v.nq * es);
    const int64_t cap = (44 * 1024 - fixed) / (8 * (v.nq + 1) * es);
    const int wr = (int)std::max<int64_t>(32, std::min(want, cap) / 32 * 32);
    const size_t smem = ((size_t)8 * wr * (v.nq + 1) + (size_t)v.nq * (MB < 4 ? 4 : MB) + (size_t)8 * 32 * ms) * sizeof(T);
    const int64_t blocks = ceil_div(v.outer, (int64_t)8 * wr);
    if (smem > 48 * 1024) {
        // staged double outputs of m up to 16 with 32-row tiles: up to 70 KB
        const cudaError_t e = cudaFuncSetAttribute(rowflat_kernel<T, MB, STAGE>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    rowflat_kernel<T, MB, STAGE><<<(unsigned)blocks, 256, smem, s>>>(v, wr);
    return cudaGetLastError();
}

// Staged (coalesced) output stores where a row's outputs take at least 64 bytes, or at least 32
// bytes with fibres of at most 4 elements (measured on A of 2^26 elements, n_q 2..16, m 4..16).
template <typename T, int MB>
cudaError_t rowflat_launch(const View3& v, cudaStream_t s)
{
    const int64_t ob = v.m * (int64_t)sizeof(T);
    const bool stage = ob >= 64 || (ob >= 32 && v.nq <= 4);
    return stage ? rowflat_launch_s<T, MB, true>(v, s) : rowflat_launch_s<T, MB, false>(v, s);
}

template <typename T, int NQ>
cudaError_t rowspan_launch(const View3& v, cudaStream_t s)
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t spans = ceil_div(v.outer, (int64_t)(64 / sizeof(T) / NQ));
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(spans, 256), (int64_t)sms * 16));
    if (v.m <= 1) rowspan_kernel<T, 1, NQ><<<blocks, 256, 0, s>>>(v);
    else if (v.m <= 2) rowspan_kernel<T, 2, NQ><<<blocks, 256, 0, s>>>(v);
    else if (v.m <= 4) rowspan_kernel<T, 4, NQ><<<blocks, 256, 0, s>>>(v);
    else if (v.m <= 8) rowspan_kernel<T, 8, NQ><<<blocks, 256, 0, s>>>(v);
    else rowspan_kernel<T, 16, NQ><<<blocks, 256, 0, s>>>(v);
    return cudaGetLastError();
}

template <int MB>
cudaError_t rowwarp_launch(const View3& v, cudaStream_t s)
{
    int sms = 0;
    const cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    constexpr int R = MB == 8 ? 4 : 8;
    const size_t smem = (size_t)MB * ceil_div(v.nq, 32) * 32 * sizeof(float);   // at most 32 KB
    const int64_t blocks = std::min<int64_t>(ceil_div(v.outer, 8 * R), (int64_t)sms * 6);
    rowwarp_kernel<MB><<<(unsigned)std::max<int64_t>(1, blocks), 256, smem, s>>>(v);
    return cudaGetLastError();
}

// Measured against the tile kernel on A of 160 MB, its time over this one's: m <= 2 1.1-1.3 from n_q =
// 33 (0.7 at 17 and 23, where lanes idle), m = 3, 4 1.06-1.1 from 99 (0.96 at 63), m = 5..8 1.05-1.07
// at 263 (1.0 at 99); 1.4-2.8 everywhere at n_q = 511 and 1023.
bool rowwarp_takes(const View3& v)
{
    return v.m <= 8 && v.nq >= (v.m <= 2 ? 32 : v.m <= 4 ? 96 : 256) && v.nq <= kRowWarpNq;
}

template <typename T>
cudaError_t rowdot_dispatch(const View3& v, cudaStream_t s, int* kid)
{
    const int64_t span = 64 / (int64_t)sizeof(T);
    const int64_t mb = v.m <= 1 ? 1 : v.m <= 2 ? 2 : v.m <= 4 ? 4 : v.m <= 8 ? 8 : 16;
    if (aligned16(v.a) && v.nq <= span && (span / v.nq) * mb * (int64_t)sizeof(T) <= 64) {
        switch (v.nq) {
        case 1: return rowspan_launch<T, 1>(v, s);
        case 2: return rowspan_launch<T, 2>(v, s);
        case 4: return rowspan_launch<T, 4>(v, s);
        case 8: return rowspan_launch<T, 8>(v, s);
        case 16: if constexpr (sizeof(T) == 4) return rowspan_launch<T, 16>(v, s); break;
        default: break;
        }
    }
    if (v.nq <= kFlatMaxNq) {
        if (v.m <= 1) return rowflat_launch<T, 1>(v, s);
        if (v.m <= 2) return rowflat_launch<T, 2>(v, s);
        if (v.m <= 4) return rowflat_launch<T, 4>(v, s);
        if (v.m <= 8) return rowflat_launch<T, 8>(v, s);
        return rowflat_launch<T, 16>(v, s);
    }
    constexpr int RV = 16 / sizeof(T);
    const bool vec = aligned16(v.a) && (v.nq % RV == 0);
    if constexpr (sizeof(T) == 4)
        if (!vec && rowwarp_takes(v)) {
            *kid = K_ROWWARP;
            return v.m <= 1 ? rowwarp_launch<1>(v, s) : v.m <= 2 ? rowwarp_launch<2>(v, s)
                 : v.m <= 4 ? rowwarp_launch<4>(v, s) : rowwarp_launch<8>(v, s);
        }
    return vec ? rowdot_dispatch_v<T, true>(v, s) : rowdot_dispatch_v<T, false>(v, s);
}

// Sum of the `parts` partial results of a split K loop, in a fixed order: c[i] = sum_z ws[z][i], in
// double (sixteen at a time), so that many parts cost no accuracy.
template <typename T>
__global__ void __launch_bounds__(256) split_reduce_kernel(const T* __restrict__ ws, int parts, int64_t n, T* __restrict__ c)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double sum = 0.0;
        for (int z0 = 0; z0 < parts; z0 += 16) {
            T x[16];   // sixteen loads in flight
#pragma unroll
            for (int z = 0; z < 16; ++z) x[z] = z0 + z < parts ? ws[(size_t)(z0 + z) * n + i] : T(0);
            double s = x[0];
#pragma unroll
            for (int z = 1; z < 16; ++z) s += x[z];
            sum += s;
        }
        c[i] = (T)sum;
    }
}

// ---------------------------------------------------------------------------------------------
// bvec: few output rows (R = outer * inner <= 8) and m <= 256: C[r][j] = sum_l A[r][l] B(j,l),
// bound by reading B (m x n_q), e.g. the order-1 product c = B a. Block b of G streams the
// contiguous l range [b lper, (b + 1) lper) of B; its partial C goes to ws[b][r][j] and
// bvec_reduce_kernel adds the G partials in a fixed order.
//   column-major B (B(j,l) = b[j + l m], the range is one contiguous block of B): thread =
//     (j vector jv of W consecutive j, l lane ls of LS); a warp's loads for one l are
//     consecutive; the LS lane partials are added in lane order at the end;
//   row-major B (B(j,l) = b[j n_q + l]): the range is cut into tiles of kBvecTile l; warp w owns
//     rows j = w, w + 8, ... and reads W consecutive l per lane (A's tile stays in L1 across the
//     rows); warp shuffles reduce, and the warp alone adds into its rows' shared partials.
// W = 16 / sizeof(T) when the vector accesses are aligned (VEC), else 1.
// ---------------------------------------------------------------------------------------------
constexpr int kBvecMaxR = 8, kBvecMaxM = 256, kBvecTile = 1024;

// Offsets in A of (row r0 + r, l = 0) for the R rows of a row tile (r = k inner + i); A's element
// (row, l) is then at offset + l inner.
template <int R>
__device__ __forceinline__ void bvec_rows(const View3& v, int64_t r0, int Rv, int64_t (&off)[R])
{
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t row = r0 + (r < Rv ? r : 0);
        const int64_t k = row / v.inner, i = row - k * v.inner;
        off[r] = k * v.nq * v.inner + i;
    }
}

// A's element (row, l), row = k inner + i
template <typename T>
__device__ __forceinline__ T bvec_a(const T* __restrict__ A, const View3& v, int64_t row, int64_t l)
{
    const int64_t k = row / v.inner, i = row - k * v.inner;
    return __ldg(A + (k * v.nq + l) * v.inner + i);
}

template <typename T, int R, bool VEC>
__global__ void __launch_bounds__(256) bvec_cm_kernel(View3 v, int64_t lper, T* __restrict__ ws)
{
    constexpr int W = VEC ? 16 / (int)sizeof(T) : 1;
    extern __shared__ __align__(16) uint8_t bvec_smem[];
    T* red = reinterpret_cast<T*>(bvec_smem);                 // [LS][R][m]
    const T* __restrict__ A = static_cast<const T*>(v.a);
    const T* __restrict__ B = static_cast<const T*>(v.b);
    const int64_t m = v.m;
    const int JV = (int)((m + W - 1) / W), LS = 256 / JV;
    const int tid = threadIdx.x, jv = tid % JV, ls = tid / JV;
    const int64_t l0 = (int64_t)blockIdx.x * lper, l1 = l0 + lper < v.nq ? l0 + lper : v.nq;
    // rows r0 .. r0 + R - 1 of this block's row tile (blockIdx.y), Rv of them in A
    const int64_t r0 = (int64_t)blockIdx.y * R, rrem = v.outer * v.inner - r0;
    const int Rv = (int)(rrem < R ? rrem : R);
    int64_t aoff[R];
    bvec_rows<R>(v, r0, Rv, aoff);
    T acc[W][R];
#pragma unroll
    for (int w = 0; w < W; ++w)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[w][r] = T(0);
    if (ls < LS) {
#pragma unroll 4
        for (int64_t l = l0 + ls; l < l1; l += LS) {
            T a[R];
#pragma unroll
            for (int r = 0; r < R; ++r) a[r] = r < Rv ? __ldg(A + aoff[r] + l * v.inner) : T(0);
            T b[W];
            const T* bp = B + l * m + (int64_t)jv * W;
            if constexpr (VEC) {
                typedef typename V16<T>::type VT;
                const VT x = __ldg(reinterpret_cast<const VT*>(bp));
#pragma unroll
                for (int w = 0; w < W; ++w) b[w] = reinterpret_cast<const T*>(&x)[w];
            } else {
                b[0] = __ldg(bp);
            }
#pragma unroll
            for (int w = 0; w < W; ++w)
#pragma unroll
                for (int r = 0; r < R; ++r) acc[w][r] = fma_t(a[r], b[w], acc[w][r]);
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int64_t j = (int64_t)jv * W + w;
            if (j < m) {
#pragma unroll
                for (int r = 0; r < R; ++r) red[((size_t)ls * R + r) * m + j] = acc[w][r];
            }
        }
    }
    __syncthreads();
    // ws[g][row][j] over all row tiles: this block's rows start at r0
    T* wb = ws + ((size_t)blockIdx.x * gridDim.y * R + (size_t)r0) * (size_t)m;
    for (int e = tid; e < R * m; e += 256) {
        T sum = red[e];
        for (int q = 1; q < LS; ++q) sum += red[(size_t)q * R * m + e];
        wb[e] = sum;
    }
}

template <typename T, int R, bool VEC>
__global__ void __launch_bounds__(256) bvec_rm_kernel(View3 v, int64_t lper, T* __restrict__ ws)
{
    constexpr int W = VEC ? 16 / (int)sizeof(T) : 1;
    __shared__ T part[R][kBvecMaxM];
    const T* __restrict__ A = static_cast<const T*>(v.a);
    const T* __restrict__ B = static_cast<const T*>(v.b);
    const int64_t m = v.m, nq = v.nq;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t l0 = (int64_t)blockIdx.x * lper, l1 = l0 + lper < nq ? l0 + lper : nq;
    const int64_t r0 = (int64_t)blockIdx.y * R, rrem = v.outer * v.inner - r0;
    const int Rv = (int)(rrem < R ? rrem : R);
    for (int e = tid; e < R * kBvecMaxM; e += 256) part[e / kBvecMaxM][e % kBvecMaxM] = T(0);
    __syncthreads();
    for (int64_t t0 = l0; t0 < l1; t0 += kBvecTile) {
        const int64_t t1 = t0 + kBvecTile < l1 ? t0 + kBvecTile : l1;
        for (int64_t j = warp; j < m; j += 8) {
            const T* bj = B + j * nq;
            T acc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r] = T(0);
#pragma unroll 2
            for (int64_t l = t0 + (int64_t)lane * W; l < t1; l += 32 * W) {
                T b[W], a[W][R];
                if constexpr (VEC) {
                    typedef typename V16<T>::type VT;
                    const VT x = __ldg(reinterpret_cast<const VT*>(bj + l));
#pragma unroll
                    for (int w = 0; w < W; ++w) b[w] = reinterpret_cast<const T*>(&x)[w];
                    if constexpr (R == 1) {
                        // one row, inner == 1 (VEC requires it for R == 1): A's W values in one load
                        const VT y = __ldg(reinterpret_cast<const VT*>(A + l));
#pragma unroll
                        for (int w = 0; w < W; ++w) a[w][0] = reinterpret_cast<const T*>(&y)[w];
                    } else {
#pragma unroll
                        for (int w = 0; w < W; ++w)
#pragma unroll
                            for (int r = 0; r < R; ++r) a[w][r] = r < Rv ? bvec_a<T>(A, v, r0 + r, l + w) : T(0);
                    }
                } else {
                    b[0] = __ldg(bj + l);
#pragma unroll
                    for (int r = 0; r < R; ++r) a[0][r] = r < Rv ? bvec_a<T>(A, v, r0 + r, l) : T(0);
                }
#pragma unroll
                for (int w = 0; w < W; ++w)
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[r] = fma_t(a[w][r], b[w], acc[r]);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
            }
            if (lane == 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) part[r][j] += acc[r];
            }
        }
    }
    __syncthreads();
    T* wb = ws + ((size_t)blockIdx.x * gridDim.y * R + (size_t)r0) * (size_t)m;
    for (int e = tid; e < R * m; e += 256) wb[e] = part[e / m][e % m];
}

// ws[g][r][j] -> C[k][j][i] (r = k inner + i): sum over the G block partials in block order.
template <typename T>
__global__ void __launch_bounds__(256) bvec_reduce_kernel(const T* __restrict__ ws, int G, View3 v, int R)
{
    T* C = static_cast<T*>(v.c);
    const int64_t n = (int64_t)R * v.m;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / v.m, j = e - r * v.m;
        if (r >= v.outer * v.inner) continue;
        T sum = T(0);
        for (int g = 0; g < G; ++g) sum += ws[(size_t)g * n + e];
        const int64_t k = r / v.inner, i = r - k * v.inner;
        C[(k * v.m + j) * v.inner + i] = sum;
    }
}

template <typename T, int R>
cudaError_t bvec_launch_r(const View3& v, dim3 G, int64_t lper, bool vec, T* ws, cudaStream_t s)
{
    if (v.b_cm) {
        constexpr int WV = 16 / (int)sizeof(T);
        const int W = vec ? WV : 1;
        const int JV = (int)((v.m + W - 1) / W), LS = 256 / JV;
        const size_t smem = (size_t)LS * R * v.m * sizeof(T);
        if (vec) bvec_cm_kernel<T, R, true><<<G, 256, smem, s>>>(v, lper, ws);
        else bvec_cm_kernel<T, R, false><<<G, 256, smem, s>>>(v, lper, ws);
    } else {
        if (vec) bvec_rm_kernel<T, R, true><<<G, 256, 0, s>>>(v, lper, ws);
        else bvec_rm_kernel<T, R, false><<<G, 256, 0, s>>>(v, lper, ws);
    }
    return cudaGetLastError();
}

template <typename T>
cudaError_t bvec_dispatch(const View3& v, int sms, cudaStream_t s, int* launches)
{
    constexpr int WV = 16 / (int)sizeof(T);
    const int64_t R = v.outer * v.inner;
    const int Rt = R <= 1 ? 1 : R <= 2 ? 2 : R <= 4 ? 4 : 8;
    // more than 8 rows (small m only): row tiles of 8 along the grid's y dimension
    const int64_t ty = ceil_div(R, Rt);
    // 16-byte accesses: B's j vectors (column-major) or l vectors (row-major; for one row also A's)
    bool vec = aligned16(v.b) && (v.b_cm ? v.m % WV == 0 : v.nq % WV == 0);
    if (!v.b_cm && Rt == 1) vec = vec && v.inner == 1 && aligned16(v.a);
    // contiguous l ranges of at least 4096 l, eight blocks per SM at most; starts on vector boundaries
    // (with row tiles: about eight blocks per SM over all tiles, l ranges of at least 1024 l)
    const int G = ty == 1 ? (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(v.nq, 4096), (int64_t)sms * 8))
                          : (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(v.nq, 1024), ceil_div((int64_t)sms * 8, ty)));
    const int64_t lper = ceil_div(ceil_div(v.nq, G), WV) * WV;
    const int Gr = (int)ceil_div(v.nq, lper);
    T* ws = nullptr;
    cudaError_t e = dev_malloc_async(reinterpret_cast<void**>(&ws), (size_t)Gr * ty * Rt * v.m * sizeof(T), s);
    if (e != cudaSuccess) return e;
    const dim3 grid((unsigned)Gr, (unsigned)ty);
    switch (Rt) {
    case 1: e = bvec_launch_r<T, 1>(v, grid, lper, vec, ws, s); break;
    case 2: e = bvec_launch_r<T, 2>(v, grid, lper, vec, ws, s); break;
    case 4: e = bvec_launch_r<T, 4>(v, grid, lper, vec, ws, s); break;
    default: e = bvec_launch_r<T, 8>(v, grid, lper, vec, ws, s); break;
    }
    if (e == cudaSuccess) {
        const int64_t n = ty * Rt * v.m;
        bvec_reduce_kernel<T><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), 1024)), 256, 0, s>>>(
            ws, Gr, v, (int)(ty * Rt));
        e = cudaGetLastError();
    }
    cudaFreeAsync(ws, s);
    if (launches) *launches = 2;
    return e;
}

constexpr int64_t kMaxSplit = 256, kSplitChainF32 = 1024;

// Parts of the K loop for a slice-GEMM whose tiles cannot fill the GPU (1 when none is needed).
// `force` (a tuner's schedule): split whenever n_q >= 2048, into enough parts for two rounds of
// blocks.
template <typename T>
int gemm_split_parts(const View3& v, int sms, int64_t& lper, bool force = false)
{
    // (float: counted in tiles of 128 columns, for parts, and so chains, no longer than those of the 128 x
    // 128 tiles before)
    constexpr int64_t BM = 128, BN = sizeof(T) == 4 ? 128 : 64, BK = 16;
    const int64_t tiles = ceil_div(v.outer * v.inner, BM) * ceil_div(v.m, BN);
    const int64_t slots = (int64_t)sms * 2;
    lper = v.nq;
    if (v.nq < 2048 || (!force && tiles * 2 > slots)) return 1;
    int64_t S = std::min<int64_t>(ceil_div(slots, tiles), v.nq / 1024);
    if (force) S = std::max<int64_t>(2, std::min<int64_t>(ceil_div(2 * slots, tiles), v.nq / 1024));
    if (sizeof(T) == 4 && v.m <= kSmallM) S = std::max<int64_t>(S, ceil_div(v.nq, kSplitChainF32));
    S = std::min<int64_t>(S, kMaxSplit);
    // workspace of S partial results at most 1 GiB
    const int64_t nc = v.outer * v.m * v.inner;
    while (S > 1 && S * nc * (int64_t)sizeof(T) > (int64_t(1) << 30)) --S;
    if (S <= 1) return 1;
    lper = ceil_div(ceil_div(v.nq, S), BK) * BK;
    return (int)ceil_div(v.nq, lper);
}

template <typename T>
cudaError_t simt_gemm_launch(const View3& v, cudaStream_t s, int* launches, bool force, bool may_split, void* space)
{
    int sms = 0;
    cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    int64_t lper = 0;
    const int S = may_split ? gemm_split_parts<T>(v, sms, lper, force) : 1;
    if (launches) *launches = S > 1 ? 2 : 1;
    if (S <= 1) return simt_gemm_dispatch(v, s, 1, 0, static_cast<T*>(nullptr));
    const int64_t nc = v.outer * v.m * v.inner;
    T* ws = static_cast<T*>(space);
    if (!space && (e = split_malloc_async(reinterpret_cast<void**>(&ws), (size_t)S * nc * sizeof(T), s)) != cudaSuccess)
        return e;
    e = simt_gemm_dispatch(v, s, S, lper, ws);
    if (e == cudaSuccess) {
        split_reduce_kernel<T><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(nc, 256), 4096)), 256, 0, s>>>(
            ws, S, nc, static_cast<T*>(v.c));
        e = cudaGetLastError();
    }
    if (!space) cudaFreeAsync(ws, s);
    return e;
}

}  // namespace

cudaError_t launch_simt_gemm(const View3& v, int dtype, cudaStream_t s, int* launches, bool force_split, bool may_split,
                             void* space)
{
    return dtype == 0 ? simt_gemm_launch<float>(v, s, launches, force_split, may_split, space)
                      : simt_gemm_launch<double>(v, s, launches, force_split, may_split, space);
}

size_t simt_gemm_split_bytes(const View3& v, int dtype)
{
    int sms = 0;
    if (sms_of_device(sms) != cudaSuccess) return 0;
    int64_t lper = 0;
    const int S = dtype == 0 ? gemm_split_parts<float>(v, sms, lper, true) : gemm_split_parts<double>(v, sms, lper, true);
    return S > 1 ? (size_t)S * (size_t)(v.outer * v.m * v.inner) * (dtype == 0 ? sizeof(float) : sizeof(double)) : 0;
}

// Measured over A of 2^14 to 2^26 elements, n_q 3 to 2001, inner 1 to 1001, as time of the small-m
// kernel over time of the slice-GEMM tile of that width.
//   double
//   m 9..16   1.1-2.8 from n_q = 12 on (0.7-1.0 at n_q = 8; fibres of at most 16 keep their
//             kernels); rows of i off 16-byte boundaries 1.3-3.6 from n_q = 64, 0.95-1.07 at 24
//   m 5..8    1.1-1.6 from n_q = 250, 0.85-1.2 at 64
//   m <= 4    1.0-1.7 from n_q = 250 where the TMA-fed kernel does not take the problem; where it
//             does, that kernel reads A at the copy rate already
//   float
//   m 9..16   rows of i 1.0-3.2 from n_q = 64 on (0.65-1.2 at 24, and 0.9 with rows of 8 elements);
//             contiguous fibres on 16-byte boundaries 1.05-1.4 from n_q = 64, off them 1.4-10 at
//             n_q = 2001 and 0.93-2.0 at 250
//   m <= 8    mostly 0.6-1.1
// Few row tiles leave the GPU idle. From n_q = 2048 on the l range is then split over more blocks
// (two launches) where the tiles come to less than 1.7 blocks an SM, as time of the kernel otherwise
// taken over time of the split tile, A of 2^21 elements and more:
//   l-split kernels (long fibres, very long strided ranges): 1.4-3.5 from 32 to 2048 rows, 3.6-25
//             beyond, any m; of unsplit tiles with n_q 1024-2047 2.2-6 from 16 tiles on
//   TMA-fed kernels, m 9..16: 1.0-1.5 float, 1.3-3.2 double (unsplit 0.3-0.9), fibres of double m 5..8
//             1.0-1.3; at most 128 rows leave its stages of 512 fibres empty: 1.4-12 (float, m 5..8
//             1.3 at 512 rows)
//   column kernel: double m 5..8 3.4-6, float m 9..16 2.1-5.4; m below that, to 8192 rows 1.7-4
// Float keeps to ranges whose parts are at most kSplitChainF32 l long, and splits whatever the block
// count in place of the l-split kernels. (The parts' sums are folded: no further off than those kernels',
// gemm_f32.cuh.)
// Shorter ranges of few tiles keep to the TMA-fed kernel (m 9..16: 0.5-0.8 at 64 blocks, 1.1 at 128; m
// 5..8 0.9 at 128, 1.1 at 256), or to the l-split kernels and the column kernel's l split (0.8-0.9
// below about 16 tiles of 128 rows).
SmallGemm small_m_takes_gemm(const View3& v, int dtype, bool tma, bool may_split)
{
    int sms = 0;
    if (sms_of_device(sms) != cudaSuccess) return SmallGemm::No;
    const int64_t rows = v.outer * v.inner, tiles = ceil_div(rows, kGemmRows);
    const bool f64 = dtype != 0, fibres = v.inner == 1;
    const bool vec = aligned16(v.a) && (fibres ? v.nq : v.inner) % (f64 ? 2 : 4) == 0;
    const int64_t blocks = ceil_div(rows, f64 && vec ? kGemmRows / 2 : kGemmRows);
    const bool lsplit = !tma && bvec_small_supported(v);   // the l-split kernels would take it
    const bool few = 10 * blocks < 17 * sms;
    if (may_split && (few || (lsplit && !f64)) && v.nq >= 2048 && (f64 || v.nq <= kSplitChainF32 * kMaxSplit) && rows > kBvecMaxR &&
        rows * v.nq >= (int64_t(1) << 21)) {
        bool take = lsplit;
        if (fibres) take = take || v.m > (f64 ? 4 : 8) || rows <= (v.m > 4 ? 4 : 1) * kGemmRows;
        else if (f64) take = take || v.m > 8 || (!tma && (v.m > 4 || tiles <= 64));
        else take = take || (v.inner >= 64 && (v.m > 8 || (!tma && tiles <= 64)));
        if (take) return SmallGemm::Split;
    }
    // ranges too long for parts of kSplitChainF32: one block per tile would leave most SMs idle
    if (lsplit && !f64 && v.nq >= 2048) return SmallGemm::No;
    if (tma && (v.m > 8 ? 20 * blocks < 17 * sms : few)) return SmallGemm::No;
    bool take;
    if (dtype == 0) {
        if (v.m <= 8) take = lsplit && tiles >= 16;
        else if (v.inner == 1) take = v.nq >= (vec ? 64 : 512) && (v.nq < 1024 || tiles >= 16);
        else take = tiles >= 32 && v.nq >= 64 && v.inner >= 64;
    } else if (v.inner == 1) {
        take = v.nq > (v.m > 8 ? kFlatMaxNq : 127) && (v.nq < 1024 || tiles >= 16) && (v.m > 4 || !tma);
    } else if (v.m > 8) {
        take = tiles >= 16 && v.nq >= (vec ? 12 : 32);
    } else {
        take = tiles >= 128 && v.nq >= 128 && (v.m > 4 || !vec);
    }
    return take ? SmallGemm::Whole : SmallGemm::No;
}

int simt_gemm_launch_count(const View3& v, int dtype)
{
    int sms = 0;
    if (sms_of_device(sms) != cudaSuccess) return 1;
    int64_t lper = 0;
    const int S = dtype == 0 ? gemm_split_parts<float>(v, sms, lper) : gemm_split_parts<double>(v, sms, lper);
    return S > 1 ? 2 : 1;
}

bool bvec_supported(const View3& v)
{
    return v.m > kSmallM && v.m <= kBvecMaxM && v.outer * v.inner <= kBvecMaxR && v.nq >= 4096;
}

bool bvec_small_supported(const View3& v)
{
    const int64_t R = v.outer * v.inner;
    if (v.m < 1 || v.m > kSmallM) return false;
    if (R <= kBvecMaxR) return v.nq >= 4096;
    // row tiles: rows too few for the column and row kernels to fill the GPU, l long enough to
    // split (measured at m = 8, 16-4095 rows: against the row kernel from n_q = 1024 on, against
    // the column kernel's l-split form only for long l ranges)
    return R <= kBvecSmallMaxRows && v.nq >= (v.inner == 1 ? 1024 : 16384);
}

cudaError_t launch_bvec(const View3& v, int dtype, cudaStream_t s, int* launches)
{
    int sms = 0;
    cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    return dtype == 0 ? bvec_dispatch<float>(v, sms, s, launches) : bvec_dispatch<double>(v, sms, s, launches);
}

// Few rows (fewer than ~32 warps of rows per SM): the l loop is split across warps.
bool colvec_splits(const View3& v, int dtype)
{
    if (dtype == 0 && few_columns_takes(v)) return false;
    const int64_t w = dtype == 0 ? colvec_rows_per_lane<float>(v) : colvec_rows_per_lane<double>(v);
    return ceil_div(v.outer * v.inner, 32 * w) < kColSplitWarps;
}

cudaError_t launch_colvec(const View3& v, int dtype, cudaStream_t s, int* kid)
{
    return launch_colvec_ls(v, dtype, colvec_splits(v, dtype) ? 8 : 1, s, kid);
}

cudaError_t launch_colvec_ls(const View3& v, int dtype, int ls, cudaStream_t s, int* kid)
{
    if (dtype == 0 && ls == 1 && few_columns_takes(v)) {
        *kid = K_FEW_COLUMNS;
        return few_columns_dispatch(v, s);
    }
    *kid = K_COLVEC;
    return dtype == 0 ? colvec_dispatch<float>(v, ls, s) : colvec_dispatch<double>(v, ls, s);
}

cudaError_t launch_rowdot(const View3& v, int dtype, cudaStream_t s, int* kid)
{
    *kid = K_ROWDOT;
    return dtype == 0 ? rowdot_dispatch<float>(v, s, kid) : rowdot_dispatch<double>(v, s, kid);
}

void grouped_columns(int64_t m, int dtype, int64_t* tiles, int* cols)
{
    ColumnGrid g = split_columns(m, kGroupNF);
    if (dtype == 0) g.nf = g.nf <= 4 ? 4 : g.nf <= 6 ? 6 : 8;   // the widths the FP32 tile is built for there
    *tiles = ceil_div(m, g.nf * 8);
    *cols = g.nf * 8;
}

int grouped_blocks_per_sm(int dtype)
{
    int n = 0;
    cudaError_t e = dtype == 0 ? cudaFuncSetAttribute(grouped_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)grouped_smem_bytes<float>())
                               : cudaFuncSetAttribute(grouped_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)grouped_smem_bytes<double>());
    if (e == cudaSuccess)
        e = dtype == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grouped_kernel<float>, 256,
                                                                       grouped_smem_bytes<float>())
                       : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grouped_kernel<double>, 256,
                                                                       grouped_smem_bytes<double>());
    return (e == cudaSuccess && n > 0) ? n : 1;
}

cudaError_t launch_grouped(const GroupDesc* d_desc, int count, int64_t total, unsigned long long* queue, int dtype,
                           int grid, cudaStream_t s)
{
    if (dtype == 0) grouped_kernel<float><<<grid, 256, grouped_smem_bytes<float>(), s>>>(d_desc, count, total, queue);
    else grouped_kernel<double><<<grid, 256, grouped_smem_bytes<double>(), s>>>(d_desc, count, total, queue);
    return cudaGetLastError();
}

int grouped_small_blocks_per_sm(int dtype)
{
    int n = 0;
    cudaError_t e = dtype == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grouped_small_kernel<float>, 256, 0)
                               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, grouped_small_kernel<double>, 256, 0);
    return (e == cudaSuccess && n > 0) ? n : 1;
}

cudaError_t launch_grouped_small(const GroupDesc* d_desc, int count, int64_t total, unsigned long long* queue,
                                 int dtype, int grid, cudaStream_t s)
{
    if (dtype == 0) grouped_small_kernel<float><<<grid, 256, 0, s>>>(d_desc, count, total, queue);
    else grouped_small_kernel<double><<<grid, 256, 0, s>>>(d_desc, count, total, queue);
    return cudaGetLastError();
}

cudaError_t launch_strided(const StridedProblem& sp, int dtype, cudaStream_t s)
{
    int64_t blocks = ceil_div(sp.total, 256);
    if (blocks > 148 * 64) blocks = 148 * 64;
    if (blocks < 1) blocks = 1;
    if (dtype == 0) strided_kernel<float><<<(unsigned)blocks, 256, 0, s>>>(sp);
    else strided_kernel<double><<<(unsigned)blocks, 256, 0, s>>>(sp);
    return cudaGetLastError();
}

template <class T>
__global__ void __launch_bounds__(256) fill_kernel(T* __restrict__ p, int64_t n, T v)
{
    const int64_t step = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step) p[i] = v;
}

cudaError_t launch_fill(void* p, int64_t n, int dtype, double v, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    int sms = 148;
    cudaError_t e = sms_of_device(sms);
    if (e != cudaSuccess) return e;
    const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), int64_t(sms) * 8);
    if (dtype == 0) fill_kernel<float><<<(unsigned)blocks, 256, 0, s>>>(static_cast<float*>(p), n, float(v));
    else fill_kernel<double><<<(unsigned)blocks, 256, 0, s>>>(static_cast<double*>(p), n, v);
    return cudaGetLastError();
}

}  // namespace tlibttm
