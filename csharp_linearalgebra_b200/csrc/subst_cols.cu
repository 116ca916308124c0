// Triangular substitution in the reference's order, one launch per solve.
//
// Per right-hand side column the reference computes
//   lower:  x[i] += (-x[k]) * L[i,k],                 k = 0..n-1, i > k
//           (after x[k] /= L[k,k] when the diagonal is explicit)
//   upper:  x[k] /= U[k,k]; x[i] += (-x[k]) * U[i,k], k = n-1..0, i < k
// with two roundings per real product and sum, skipping the updates of a zero
// x[k] (Triangular.SolveLowerUnit / SolveLower / SolveUpper, BlockedLu.cs:312-352;
// complex divisions are skipped for a zero x[k] too). Each x[i] is one chain in
// the order of k, and columns never meet, so a CTA can own a few columns and
// run the whole solve on them without another CTA: the columns sit in shared
// memory, the interchanges are applied as they are read, and both triangles
// run in one launch. (One launch per 32-row block for the triangle and one for
// the rows beyond it took 62 launches at n = 512, 2.4 ms for 512 complex
// columns, most of it in the triangles' kernel, whose unrolled body missed the
// instruction cache.)
//
// Blocks of 32 rows, in the order of k, in phases of one block barrier each.
// In phase p, four warps finish block p + 1 while eight update the rows
// beyond it with block p:
//   triangle  a warp per column or two, a row per lane: first block p's steps
//             reach the rows of block p + 1 (that 32 x 32 piece of the factor
//             staged in shared memory), then step k of the triangle broadcasts
//             x[k] by shuffles and every later lane continues its chain. The
//             diagonal divisions use the divisor's reciprocal, prepared once per
//             block (divide.cuh): 40 cycles in the chain for a division's 113.
//   update    a warp takes 32 rows (64 real) of all C columns, a row (two) and
//             its C values per thread in registers, block p's solved x
//             broadcast from shared memory, the factor's columns read from L2
//             once per CTA (consecutive lanes, consecutive rows), the next
//             steps' entries in flight while these are applied.

#include "subst_cols.h"

#include <algorithm>
#include <atomic>
#include <climits>

#include "batch.cuh"
#include "device_util.cuh"
#include "divide.cuh"

namespace tns {

namespace {

constexpr int kB = kDiagBlock;    // rows per block
constexpr int kTriWarps = 4;      // warps that solve the triangles
constexpr int kUpdWarps = 8;      // warps that update the rows beyond
constexpr int kThreads = 32 * (kTriWarps + kUpdWarps);

struct ColsDesc {
    SubstCols s;
    int tile_begin;  // this item's first CTA
};

template <bool CPLX>
struct El;
template <>
struct El<false> {
    using T = double;
    // in integers, off the FP64 pipe
    static __device__ __forceinline__ bool zero(double v) { return (__double_as_longlong(v) << 1) == 0; }
    static __device__ __forceinline__ double neg(double v) { return -v; }
    static __device__ __forceinline__ double axpy(double x, double nxk, double f) { return add_rn(x, mul_rn(nxk, f)); }
    static __device__ __forceinline__ double shfl(double v, int k) { return __shfl_sync(0xffffffffu, v, k); }
};
template <>
struct El<true> {
    using T = double2;
    static __device__ __forceinline__ bool zero(double2 v) {
        return ((__double_as_longlong(v.x) | __double_as_longlong(v.y)) << 1) == 0;
    }
    static __device__ __forceinline__ double2 neg(double2 v) { return make_double2(-v.x, -v.y); }
    static __device__ __forceinline__ double2 axpy(double2 x, double2 a, double2 b) {
        const double re = sub_rn(mul_rn(a.x, b.x), mul_rn(a.y, b.y));
        const double im = add_rn(mul_rn(a.y, b.x), mul_rn(a.x, b.y));
        return make_double2(add_rn(x.x, re), add_rn(x.y, im));
    }
    static __device__ __forceinline__ double2 shfl(double2 v, int k) {
        return make_double2(__shfl_sync(0xffffffffu, v.x, k), __shfl_sync(0xffffffffu, v.y, k));
    }
};

__device__ __forceinline__ void cp_async(double2* dst, const double2* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

// Shared memory of a CTA with C columns of order n.
template <bool CPLX, int C>
struct Layout {
    using E = typename El<CPLX>::T;
    static constexpr int kTile = kB * kB;
    // the columns, two triangles and the pieces beside them, two blocks of
    // negated solutions, each triangle warp's divisors
    static size_t bytes(int n) {
        return sizeof(E) * ((size_t)C * n + 4 * kTile + 2 * kB * C) + sizeof(Divisor) * kB * kTriWarps;
    }
};

// C consecutive entries of shared memory, by 16-byte loads.
template <int C>
__device__ __forceinline__ void load_row(const double2* p, double2 (&v)[C]) {
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = p[c];
}
template <int C>
__device__ __forceinline__ void load_row(const double* p, double (&v)[C]) {
    if constexpr (C == 1) {
        v[0] = p[0];
    } else {
#pragma unroll
        for (int c = 0; c < C; c += 2) {
            const double2 t = *reinterpret_cast<const double2*>(p + c);
            v[c] = t.x;
            v[c + 1] = t.y;
        }
    }
}

// Rows [r0, r1) take the steps of block [k0, k0 + kB), by the update warps
// (warp 0..kUpdWarps - 1), for the C columns in xs, from the negated solved values xb[k * C + c]. CHECKED: some
// of them are zero (their updates are skipped) or the block is short (its
// missing steps are zeros, and their factor columns are not read).
template <bool CPLX, bool UPPER, int C, bool CHECKED>
__device__ __forceinline__ void update_rows(const typename El<CPLX>::T* __restrict__ f, int ldf,
                                            typename El<CPLX>::T* xs, int n, const typename El<CPLX>::T* xb, int k0,
                                            int w, int r0, int r1, int warp) {
    using El_ = El<CPLX>;
    using E = typename El_::T;
    constexpr int R = CPLX ? 1 : 2;      // rows per thread, every column
    constexpr int G = CPLX && C == 8 ? 2 : C >= 4 ? 4 : 8;  // steps whose factor entries are loaded together
    const int lane = threadIdx.x & 31;
    const int chunks = (r1 - r0 + 32 * R - 1) / (32 * R);
    for (int t = warp; t < chunks; t += kUpdWarps) {
        const int i0 = r0 + t * 32 * R + lane;
        bool ok[R];
        E acc[R][C];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            ok[r] = i0 + 32 * r < r1;
#pragma unroll
            for (int c = 0; c < C; ++c) acc[r][c] = ok[r] ? xs[(size_t)c * n + i0 + 32 * r] : E{};
        }
        const E* fp = f + (size_t)k0 * ldf + i0;
        E fv[2][G][R];
        auto load = [&](int g, E (&v)[G][R]) {
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const int s = g * G + j, k = UPPER ? kB - 1 - s : s;
#pragma unroll
                for (int r = 0; r < R; ++r)
                    v[j][r] = ok[r] && (!CHECKED || k < w) ? fp[(size_t)k * ldf + 32 * r] : E{};
            }
        };
        auto apply = [&](int g, const E (&v)[G][R]) {
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const int s = g * G + j, k = UPPER ? kB - 1 - s : s;
                E nx[C];
                load_row<C>(xb + k * C, nx);
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    if (CHECKED && El_::zero(nx[c])) continue;
#pragma unroll
                    for (int r = 0; r < R; ++r) acc[r][c] = El_::axpy(acc[r][c], nx[c], v[j][r]);
                }
            }
        };
        load(0, fv[0]);
#pragma unroll 1
        for (int g = 0; g < kB / G; g += 2) {
            load(g + 1, fv[1]);
            apply(g, fv[0]);
            if (g + 2 < kB / G) load(g + 2, fv[0]);
            apply(g + 1, fv[1]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (ok[r]) xs[(size_t)c * n + i0 + 32 * r] = acc[r][c];
    }
}

__device__ __forceinline__ double pick(bool c, double a, double b) { return c ? a : b; }
__device__ __forceinline__ double2 pick(bool c, double2 a, double2 b) {
    return make_double2(c ? a.x : b.x, c ? a.y : b.y);
}

// The steps of one block's own triangle t (t[k * kB + i] = F[k0 + i, k0 + k], w
// rows) for a warp's NQ columns, row `lane` of each in v. FAST: the prepared
// reciprocals throughout; false when a dividend was out of their range (v is
// then meaningless). The step is one dependent chain, so its conditions are
// selects: a branch in it measured 127 cycles a unit lower complex step
// against 81.
template <bool CPLX, bool UPPER, bool DIV, int NQ, bool FAST>
__device__ __forceinline__ bool triangle_steps(const typename El<CPLX>::T* t, int w, typename El<CPLX>::T (&v)[NQ],
                                               const Divisor* dv) {
    using El_ = El<CPLX>;
    using E = typename El_::T;
    const int lane = threadIdx.x & 31;
    bool good = true;
#pragma unroll 4
    for (int step = 0; step < w; ++step) {
        const int k = UPPER ? w - 1 - step : step;
        const E tk = t[k * kB + lane];  // (rows past w are not used)
        const bool later = UPPER ? lane < k : lane > k;
        E x[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) x[q] = El_::shfl(v[q], k);
        if constexpr (UPPER || DIV) {
            const Divisor d = dv[k];
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if constexpr (FAST) {
                    good = divide_fast(x[q], d, x[q]) & good;
                } else {
                    // Always for real; for complex when x_k is not zero.
                    if (!CPLX || !El_::zero(x[q])) x[q] = divide(x[q], d);
                }
                v[q] = pick(lane == k, x[q], v[q]);
            }
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const E next = El_::axpy(v[q], El_::neg(x[q]), tk);
            v[q] = pick(later & !El_::zero(x[q]), next, v[q]);
        }
    }
    return good;
}

template <bool CPLX, bool UPPER, bool DIV, int NQ>
__device__ __forceinline__ void triangle(const typename El<CPLX>::T* t, int w, typename El<CPLX>::T (&v)[NQ],
                                         Divisor* dv) {
    using E = typename El<CPLX>::T;
    if constexpr (UPPER || DIV) {
        const int lane = threadIdx.x & 31;
        Divisor mine{};
        mine.safe = 1;
        if (lane < w) mine = make_divisor(t[lane * kB + lane]);
        dv[lane] = mine;
        __syncwarp();  // a vote orders no memory
        const bool all_safe = __all_sync(0xffffffffu, mine.safe);
        E kept[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) kept[q] = v[q];
        // The dividends are the same in every lane, and so is the answer.
        if (all_safe && triangle_steps<CPLX, UPPER, DIV, NQ, true>(t, w, v, dv)) return;
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = kept[q];
    }
    triangle_steps<CPLX, UPPER, DIV, NQ, false>(t, w, v, dv);
}

// One triangle: UPPER (explicit diagonal) or lower (DIV: explicit diagonal,
// else unit).
template <bool CPLX, bool UPPER, bool DIV, int C>
__device__ void solve_triangle(const SubstCols& s, typename El<CPLX>::T* xs, typename El<CPLX>::T* tiles,
                               typename El<CPLX>::T* xb, Divisor* divs, int* s_zero) {
    using El_ = El<CPLX>;
    using E = typename El_::T;
    constexpr int NQ = C > kTriWarps ? C / kTriWarps : 1;  // columns of a triangle warp
    constexpr int kTile = kB * kB;
    const int n = s.n, ldf = s.ldf;
    const E* f = reinterpret_cast<const E*>(s.f);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int blocks = (n + kB - 1) / kB;
    auto block = [&](int p) { return UPPER ? blocks - 1 - p : p; };  // the p-th block solved
    // For the p-th block: its triangle, and the piece of the factor that takes
    // the block before it to its rows, into the buffers of parity p & 1.
    auto stage = [&](int p) {
        if (p < blocks) {
            const int k0 = block(p) * kB, w = min(kB, n - k0);
            E* t = tiles + (p & 1) * 2 * kTile;
            const int j0 = p > 0 ? block(p - 1) * kB : 0, wj = p > 0 ? min(kB, n - j0) : 0;
            for (int e = threadIdx.x; e < 2 * kTile; e += kThreads) {
                const int k = (e % kTile) / kB, i = e % kB;
                if (e < kTile) {
                    if (i < w && k < w) cp_async(t + e, f + (size_t)(k0 + k) * ldf + k0 + i);
                } else if (i < w && k < wj) {
                    cp_async(t + e, f + (size_t)(j0 + k) * ldf + k0 + i);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0);
    stage(1);
    // Phase p: the triangle warps finish block p + 1, the others take block p
    // to the rows beyond it. Phase -1 solves the first block.
    for (int p = -1; p < blocks - 1; ++p) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (threadIdx.x == 0) s_zero[(p + 1) & 1] = 0;  // block p + 1's flag; block p - 1's readers are past
        __syncthreads();
        if (warp < kTriWarps) {
            if (warp * NQ < C) {
                const int q1 = p + 1, k0 = block(q1) * kB, w = min(kB, n - k0);
                const E* t = tiles + (q1 & 1) * 2 * kTile;
                const E* side = t + kTile;
                E v[NQ];
#pragma unroll
                for (int q = 0; q < NQ; ++q) v[q] = lane < w ? xs[(size_t)(warp * NQ + q) * n + k0 + lane] : E{};
                if (p >= 0) {
                    const int wj = min(kB, n - block(p) * kB);
                    const E* xp = xb + (p & 1) * kB * C + warp * NQ;
                    const bool checked = s_zero[p & 1];
#pragma unroll 8
                    for (int step = 0; step < wj; ++step) {
                        const int k = UPPER ? wj - 1 - step : step;
                        const E fk = side[k * kB + lane];
#pragma unroll
                        for (int q = 0; q < NQ; ++q) {
                            const E nx = xp[k * C + q];
                            if (!checked || !El_::zero(nx)) v[q] = El_::axpy(v[q], nx, fk);
                        }
                    }
                }
                triangle<CPLX, UPPER, DIV, NQ>(t, w, v, divs + warp * kB);
                E* xn = xb + (q1 & 1) * kB * C + warp * NQ;
                bool zero = w < kB;  // a short block's missing steps are zeros
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    if (lane < w) xs[(size_t)(warp * NQ + q) * n + k0 + lane] = v[q];
                    xn[lane * C + q] = lane < w ? El_::neg(v[q]) : E{};
                    zero = zero || El_::zero(v[q]);
                }
                if (zero) s_zero[q1 & 1] = 1;
            }
        } else if (p >= 0) {
            const int k0 = block(p) * kB, w = min(kB, n - k0);
            const int r0 = UPPER ? 0 : k0 + 2 * kB, r1 = UPPER ? k0 - kB : n;
            const E* xp = xb + (p & 1) * kB * C;
            if (r1 > r0) {
                if (s_zero[p & 1])
                    update_rows<CPLX, UPPER, C, true>(f, ldf, xs, n, xp, k0, w, r0, r1, warp - kTriWarps);
                else
                    update_rows<CPLX, UPPER, C, false>(f, ldf, xs, n, xp, k0, w, r0, r1, warp - kTriWarps);
            }
        }
        __syncthreads();
        stage(p + 3);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

template <bool CPLX, int C>
__global__ void __launch_bounds__(kThreads, 1)
    subst_cols_kernel(const __grid_constant__ Batch<ColsDesc> b, int lower, int upper) {
    using E = typename El<CPLX>::T;
    int lo = 0, hi = b.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (batch_item(b, mid).tile_begin <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const ColsDesc& d = batch_item(b, lo);
    const SubstCols s = d.s;
    const int n = s.n, col0 = ((int)blockIdx.x - d.tile_begin) * C;
    extern __shared__ __align__(16) unsigned char cols_smem[];
    __shared__ int s_zero[2];
    E* xs = reinterpret_cast<E*>(cols_smem);  // [C][n]
    E* tiles = xs + (size_t)C * n;            // [2][triangle, side][kB][kB]
    E* xb = tiles + 4 * kB * kB;              // [2][kB][C]
    Divisor* divs = reinterpret_cast<Divisor*>(xb + 2 * kB * C);
    E* x = reinterpret_cast<E*>(s.x);
    // A column past the last one is a copy of the CTA's first and is not
    // written back.
#pragma unroll 1
    for (int c = 0; c < C; ++c) {
        const E* src = x + (size_t)(col0 + c < s.nrhs ? col0 + c : col0) * s.ldx;
        for (int i = threadIdx.x; i < n; i += kThreads) xs[(size_t)c * n + i] = src[s.perm ? s.perm[i] : i];
    }
    __syncthreads();
    if (lower == (int)LowerKind::kUnit) solve_triangle<CPLX, false, false, C>(s, xs, tiles, xb, divs, s_zero);
    else if (lower == (int)LowerKind::kDivide) solve_triangle<CPLX, false, true, C>(s, xs, tiles, xb, divs, s_zero);
    if (upper) solve_triangle<CPLX, true, true, C>(s, xs, tiles, xb, divs, s_zero);
#pragma unroll 1
    for (int c = 0; c < C && col0 + c < s.nrhs; ++c) {
        E* dst = x + (size_t)(col0 + c) * s.ldx;
        for (int i = threadIdx.x; i < n; i += kThreads) dst[i] = xs[(size_t)c * n + i];
    }
}

// ---- diagonal blocks of the blocked solves -----------------------------------

// Up to eight steps with a working width of NC rows, from step s0: the step's
// row is always a[0], its solution goes back to x and the later rows shift
// down by one, so the loop has static register indices and its code (76 row
// updates over the four widths) stays in the instruction cache, which the
// same solve unrolled over 32 steps missed (70 us a launch against 7).
template <bool CPLX, bool UPPER, bool DIV, int NC>
__device__ __forceinline__ void diag_phase(const typename El<CPLX>::T* t, const Divisor* dv, bool all_safe,
                                           typename El<CPLX>::T (&a)[kB], typename El<CPLX>::T* x, bool live, int w,
                                           int s0) {
    using El_ = El<CPLX>;
    using E = typename El_::T;
    const int send = min(s0 + 8, w);
#pragma unroll 1
    for (int s = s0; s < send; ++s) {
        const int k = UPPER ? w - 1 - s : s;
        E xk = a[0];
        if constexpr (UPPER || DIV) {
            const Divisor d = dv[k];
            E y;
            const bool fast = divide_fast(xk, d, y);
            if (__all_sync(0xffffffffu, all_safe && fast)) xk = y;
            else if (!CPLX || !El_::zero(xk)) xk = divide(xk, d);
        }
        if (live) x[k] = xk;
        const bool skip = El_::zero(xk);
        const E nx = El_::neg(xk);
        const E* tk = t + k * kB + k;  // tk[+-c]: the entry of the row c steps on
        if (!__any_sync(0xffffffffu, skip)) {
#pragma unroll
            for (int c = 1; c < NC; ++c) a[c - 1] = El_::axpy(a[c], nx, tk[UPPER ? -c : c]);
        } else {
#pragma unroll
            for (int c = 1; c < NC; ++c) {
                const E next = El_::axpy(a[c], nx, tk[UPPER ? -c : c]);
                a[c - 1] = pick(skip, a[c], next);
            }
        }
    }
}

// One thread per right-hand side: every lane's arithmetic is its own column's,
// so the triangle costs the FP64 pipe nothing twice.
template <bool CPLX, bool UPPER, bool DIV>
__global__ void __launch_bounds__(128) diag_block_kernel(const __grid_constant__ Batch<SubstDiagDesc> b) {
    using E = typename El<CPLX>::T;
    const SubstDiagDesc& d = batch_item(b, blockIdx.y);
    if ((int)(blockIdx.x * blockDim.x) >= d.nrhs) return;  // the whole block
    const int w = d.w;
    // t[k * kB + i] = F[k0 + i, k0 + k], zeros past w, between two margins that
    // the rows past a block's end read (and whose results nothing uses)
    __shared__ E s_t[kB + kB * kB + kB];
    __shared__ Divisor s_dv[kB];
    E* t = s_t + kB;
    const E* f = reinterpret_cast<const E*>(d.f);
    for (int e = threadIdx.x; e < kB * kB + 2 * kB; e += blockDim.x) {
        const int k = e / kB - 1, i = e % kB;
        s_t[e] = k >= 0 && k < w && i < w ? f[(size_t)(d.k0 + k) * d.ldf + d.k0 + i] : E{};
    }
    __syncthreads();
    bool all_safe = true;
    if constexpr (UPPER || DIV) {
        if (threadIdx.x < kB) {
            Divisor mine{};
            mine.safe = 1;
            if ((int)threadIdx.x < w) mine = make_divisor(t[threadIdx.x * kB + threadIdx.x]);
            s_dv[threadIdx.x] = mine;
        }
        __syncthreads();
        all_safe = __all_sync(0xffffffffu, s_dv[threadIdx.x & 31].safe);
    }
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    // A thread past the last column works on a copy of it and writes nothing.
    const bool live = col < d.nrhs;
    E* x = reinterpret_cast<E*>(d.x) + (size_t)min(col, d.nrhs - 1) * d.ldx + d.k0;
    E a[kB];
#pragma unroll
    for (int c = 0; c < kB; ++c) a[c] = c < w ? x[UPPER ? w - 1 - c : c] : E{};
    diag_phase<CPLX, UPPER, DIV, 32>(t, s_dv, all_safe, a, x, live, w, 0);
    if (w > 8) diag_phase<CPLX, UPPER, DIV, 24>(t, s_dv, all_safe, a, x, live, w, 8);
    if (w > 16) diag_phase<CPLX, UPPER, DIV, 16>(t, s_dv, all_safe, a, x, live, w, 16);
    if (w > 24) diag_phase<CPLX, UPPER, DIV, 8>(t, s_dv, all_safe, a, x, live, w, 24);
}

template <bool CPLX>
void run_diag(Context& ctx, LowerKind lower, bool upper, const std::vector<SubstDiagDesc>& v) {
    int mr = 0;
    for (auto& d : v) mr = std::max(mr, d.nrhs);
    Batch<SubstDiagDesc> b = make_batch(ctx, v);
    const dim3 grid((mr + 127) / 128, b.count);
    if (upper) diag_block_kernel<CPLX, true, true><<<grid, 128, 0, ctx.stream>>>(b);
    else if (lower == LowerKind::kDivide) diag_block_kernel<CPLX, false, true><<<grid, 128, 0, ctx.stream>>>(b);
    else diag_block_kernel<CPLX, false, false><<<grid, 128, 0, ctx.stream>>>(b);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
}

constexpr size_t kMaxSmem = 220 * 1024;

template <bool CPLX, int C>
void launch(Context& ctx, std::vector<ColsDesc>& v, int nmax, LowerKind lower, bool upper) {
    static std::atomic<bool> configured[64];
    if (!configured[ctx.device].load(std::memory_order_acquire)) {
        TNS_CUDA(cudaFuncSetAttribute(subst_cols_kernel<CPLX, C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kMaxSmem));
        configured[ctx.device].store(true, std::memory_order_release);
    }
    long long total = 0;
    for (auto& d : v) {
        d.tile_begin = (int)total;
        total += (d.s.nrhs + C - 1) / C;
    }
    if (total > INT_MAX) fail(TNS_E_ARGUMENT, "triangular solve too large for one launch");
    subst_cols_kernel<CPLX, C><<<(unsigned)total, kThreads, Layout<CPLX, C>::bytes(nmax), ctx.stream>>>(
        make_batch(ctx, v), (int)lower, upper ? 1 : 0);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
}

// The most columns per CTA (each reads the factors once) that still give four
// SMs in five a CTA and fit shared memory; ctas(c): the CTAs of c columns.
template <bool CPLX, class F>
int columns_per_cta(const Context& ctx, int nmax, F&& ctas) {
    const long long want = ctx.num_sms * 4 / 5;
    if (ctas(8) >= want && Layout<CPLX, 8>::bytes(nmax) <= kMaxSmem) return 8;
    if (ctas(4) >= want && Layout<CPLX, 4>::bytes(nmax) <= kMaxSmem) return 4;
    if (ctas(2) >= want && Layout<CPLX, 2>::bytes(nmax) <= kMaxSmem) return 2;
    return 1;
}

template <bool CPLX>
void run(Context& ctx, LowerKind lower, bool upper, const std::vector<SubstCols>& items) {
    std::vector<ColsDesc> v;
    int nmax = 0;
    for (auto& it : items)
        if (it.n > 0 && it.nrhs > 0) {
            v.push_back(ColsDesc{it, 0});
            nmax = std::max(nmax, it.n);
        }
    if (v.empty()) return;
    // Longest solves first: the launch ends on short ones.
    std::stable_sort(v.begin(), v.end(), [](const ColsDesc& x, const ColsDesc& y) { return x.s.n > y.s.n; });
    auto ctas = [&](int c) {
        long long t = 0;
        for (auto& d : v) t += (d.s.nrhs + c - 1) / c;
        return t;
    };
    const int c = columns_per_cta<CPLX>(ctx, nmax, ctas);
    if (c == 8) launch<CPLX, 8>(ctx, v, nmax, lower, upper);
    else if (c == 4) launch<CPLX, 4>(ctx, v, nmax, lower, upper);
    else if (c == 2) launch<CPLX, 2>(ctx, v, nmax, lower, upper);
    else launch<CPLX, 1>(ctx, v, nmax, lower, upper);
}

}  // namespace

int subst_cols_max_order(bool cplx) {
    const size_t fixed = cplx ? Layout<true, 1>::bytes(0) : Layout<false, 1>::bytes(0);
    return (int)((kMaxSmem - fixed) / (cplx ? 16 : 8));
}

int subst_cols_per_cta(const Context& ctx, bool cplx, int n, long long nrhs) {
    auto ctas = [&](int c) { return (nrhs + c - 1) / c; };
    return cplx ? columns_per_cta<true>(ctx, n, ctas) : columns_per_cta<false>(ctx, n, ctas);
}

void subst_cols(Context& ctx, bool cplx, LowerKind lower, bool upper, const std::vector<SubstCols>& items) {
    if (cplx) run<true>(ctx, lower, upper, items);
    else run<false>(ctx, lower, upper, items);
}

void solve_diag_blocks(Context& ctx, bool cplx, LowerKind lower, bool upper, const std::vector<SubstDiagDesc>& v) {
    if (v.empty()) return;
    if (cplx) run_diag<true>(ctx, lower, upper, v);
    else run_diag<false>(ctx, lower, upper, v);
}

}  // namespace tns
