// Left-looking triangular solves with one chain warp per CTA and producers.
//
// The reference's transposed solves form, row by row, an inner product over the
// rows already solved, in a prescribed order:
//   U^T forward   x[i] = (x[i] - Dot(f[0..i), x[0..i))) / f_ii
//   L^T backward  x[i] -= Dot(f(i..n), x(i..n)), or divided as well
// with ColumnOps.Dot's order (ColumnOps.cs:35-65): sixteen partial sums of the
// terms of equal position modulo 16, combined pairwise, then the remaining whole
// fours, then the tail term by term (Triangular.cs:152-206); complex
//   L^H backward  x[i] = x[i] - conj(f_ki) x[k], k = i + 1 .. n - 1 in turn
//                 (BlockedLu.cs:357-373).
// Row i needs the row just before it, so a solve is one dependent chain through
// all rows. What the newest x does not enter is taken off that chain here: in
// phases of a few rows (one block barrier each), one warp solves the phase's
// rows while the other warps prepare the next phase's from the x known so far.
//   forward   the newest x come last in a row's sums, so the producers keep the
//             sixteen partial sums of the next 16 rows (a half-warp per row, up to
//             the last block but one), and the chain adds the last blocks' terms:
//             per four rows one round of partials, one combination, and then the
//             subtractions and divisions (by prepared divisors) themselves.
//   backward  the newest x come first, so no sum can run ahead, but the products
//             can: the producers write them to shared memory, and the chain
//             adds them (real: sixteen lanes of n/16 additions a row; complex:
//             one sum of n subtractions, 8 cycles each).
// The kernels these replace formed each row's products inside the chain, one
// warp per two right-hand sides: n = 512 real 434 + 443 us, n = 389 complex 792 us.

#include "subst_left.h"

#include <algorithm>
#include <atomic>

#include "device_util.cuh"
#include "divide.cuh"

namespace tns {

namespace {

constexpr int kRows = 16;                    // forward: rows per phase
constexpr int kProducers = 8;                // producer warps
constexpr int kThreads = 32 * (1 + kProducers);
constexpr size_t kMaxSmem = 220 * 1024;

// ---- real, forward -------------------------------------------------------------

struct ForwardShared {
    double acc[2][kRows][17];   // partial sums of a phase's rows, over all blocks but the last
    double in[2][kRows][17];    // in[r][k] = f[16 b + k, 16 b + r]
    double prev[2][kRows][17];  // prev[r][L] = f[16 (b - 1) + L, 16 b + r]
    Divisor div[2][kRows];
};

__device__ void forward_real(const double* __restrict__ f, int ldf, double* x, int n, ForwardShared& S) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, L = lane & 15, half = lane >> 4;
    const int blocks = (n + kRows - 1) / kRows;
    // A producer's entries of block b's two pieces (zeros past n): its row r =
    // (thread - 32) / 16 and column L of each.
    static_assert(kThreads - 32 == kRows * kRows, "one producer per entry of a piece");
    const int pr = (int)(threadIdx.x - 32) >> 4;
    auto load = [&](int b, double& in, double& prev) {
        const int i = b * kRows + pr;
        in = i < n && b * kRows + L < n ? f[(size_t)i * ldf + b * kRows + L] : 0.0;
        prev = i < n && b > 0 ? f[(size_t)i * ldf + (b - 1) * kRows + L] : 0.0;
    };
    if (warp > 0) {
        load(0, S.in[0][pr][L], S.prev[0][pr][L]);
        if (pr == L) S.div[0][L] = make_divisor(L < n ? S.in[0][L][L] : 1.0);
        S.acc[0][pr][L] = 0.0;
    }
    __syncthreads();
    for (int b = 0; b < blocks; ++b) {
        if (warp > 0) {
            // Block b + 1's rows over blocks 0 .. b - 1, a half-warp per row.
            if (b + 1 < blocks) {
                double in, prev;
                load(b + 1, in, prev);
                const int i = (b + 1) * kRows + pr;
                double acc = 0.0;
                if (i < n) {
                    const double* col = f + (size_t)i * ldf + L;
                    int q = 0;
                    for (; q + 16 <= b; q += 16) {
                        double v[16];
#pragma unroll
                        for (int u = 0; u < 16; ++u) v[u] = col[(q + u) * kRows];
#pragma unroll
                        for (int u = 0; u < 16; ++u) acc = add_rn(acc, mul_rn(v[u], x[(q + u) * kRows + L]));
                    }
                    double v[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) v[u] = q + u < b ? col[(q + u) * kRows] : 0.0;
#pragma unroll
                    for (int u = 0; u < 16; ++u)
                        if (q + u < b) acc = add_rn(acc, mul_rn(v[u], x[(q + u) * kRows + L]));
                }
                S.acc[(b + 1) & 1][pr][L] = acc;
                S.in[(b + 1) & 1][pr][L] = in;
                S.prev[(b + 1) & 1][pr][L] = prev;
                if (pr == L) S.div[(b + 1) & 1][L] = make_divisor(i < n ? in : 1.0);
            }
        } else {
            // Rows 4 g + 2 half + {0, 1} of group g: this half-warp's partials.
            const int i0 = b * kRows;
            double(&in)[kRows][17] = S.in[b & 1];
            double a[4][2];
            const double xl = b > 0 ? x[i0 - kRows + L] : 0.0;
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int r = 4 * g + 2 * half + q;
                    a[g][q] = S.acc[b & 1][r][L];
                    if (b > 0) a[g][q] = add_rn(a[g][q], mul_rn(S.prev[b & 1][r][L], xl));
                }
            const Divisor* dv = S.div[b & 1];
            double rhs[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) rhs[r] = i0 + r < n ? x[i0 + r] : 1.0;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                double t[4] = {0.0, 0.0, 0.0, 0.0};
                if (b > 0 || g > 0) {  // (a row of fewer than four terms has only a tail)
                    const double c0 = netdot_combine(a[g][0], L, lane & 16);
                    const double c1 = netdot_combine(a[g][1], L, lane & 16);
                    t[0] = __shfl_sync(0xffffffffu, c0, 0);
                    t[1] = __shfl_sync(0xffffffffu, c1, 0);
                    t[2] = __shfl_sync(0xffffffffu, c0, 16);
                    t[3] = __shfl_sync(0xffffffffu, c1, 16);
                }
                // The group's four rows: the tails, the subtractions, the divisions;
                // again with plain divisions when a dividend was out of range.
                double v[4];
                auto solve = [&](auto quotient) {
                    bool good = true;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int r = 4 * g + q;
                        double sum = t[q];
#pragma unroll
                        for (int p = 0; p < q; ++p) sum = add_rn(sum, mul_rn(in[r][4 * g + p], v[p]));
                        good = quotient(sub_rn(rhs[r], sum), dv[r], v[q]) & good;
                    }
                    return good;
                };
                if (!solve([](double a, const Divisor& d, double& y) { return divide_fast(a, d, y) & (d.safe != 0); }))
                    solve([](double a, const Divisor& d, double& y) {
                        y = __ddiv_rn(a, d.b);
                        return true;
                    });
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (lane == q && i0 + 4 * g + q < n) x[i0 + 4 * g + q] = v[q];
                // The group's four values are terms of partials 0..3 of the later rows.
                if (L < 4) {
                    const double xv = L == 0 ? v[0] : L == 1 ? v[1] : L == 2 ? v[2] : v[3];
#pragma unroll
                    for (int h = g + 1; h < 4; ++h)
#pragma unroll
                        for (int q = 0; q < 2; ++q)
                            a[h][q] = add_rn(a[h][q], mul_rn(in[4 * h + 2 * half + q][4 * g + L], xv));
                }
                __syncwarp();
            }
        }
        __syncthreads();
    }
}

// sum +- p[S m] for m in [0, count) in turn, count a positive multiple of 8: the
// next eight are loaded while eight are added. (Lists are filled up with zeros,
// which change no sum here: a sum that starts from +0 is never -0, and a
// difference keeps its sign.)
template <int S, bool ADD>
__device__ __forceinline__ double chain(double sum, const double* p, int count) {
    auto step = [](double a, double b) { return ADD ? add_rn(a, b) : sub_rn(a, b); };
    // Two sets of registers in turn: copying one to the other costs as much as
    // the additions (12 cycles a term against 8.6).
    double v[8], w[8];
    auto load = [](double (&r)[8], const double* q) {
#pragma unroll
        for (int u = 0; u < 8; ++u) r[u] = q[S * u];
    };
    auto fold = [&](const double (&r)[8]) {
#pragma unroll
        for (int u = 0; u < 8; ++u) sum = step(sum, r[u]);
    };
    load(v, p);
#pragma unroll 1
    for (; count >= 24; count -= 16) {
        load(w, p + 8 * S);
        fold(v);
        p += 16 * S;
        load(v, p);
        fold(w);
    }
    if (count > 8) load(w, p + 8 * S);
    fold(v);
    if (count > 8) fold(w);
    return sum;
}

// ---- real, backward ------------------------------------------------------------

// RB rows per phase (8, fewer for larger orders: two buffers of RB rows of
// products). A row's list in P, written by the producers: for each lane L < 16
// the products it adds after its first, entry 16 u + L being position
// m = 16 (u + 1) + L of the row (k = i + 1 + m) for the whole sixteens, then the
// whole fours of lanes 0..3, then zeros up to a multiple of eight per lane; and
// behind it the tail's up to three products. The chain forms the first sixteen
// products itself (their x are the newest). Rows of fewer than 16 terms have no
// list.
__host__ __device__ inline int list_length(int len) { return ((len >> 4) - 1 + 3 + 7) & ~7; }
__host__ __device__ inline size_t list_pitch(int n) { return 16 * (size_t)list_length(n) + 4; }

template <bool DIV, int RB>
__device__ void backward_real(const double* __restrict__ f, int ldf, double* x, int n, double* P,
                              double (*head)[RB][16], double* diag) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, L = lane & 15;
    const int blocks = (n + RB - 1) / RB;
    const size_t pitch = list_pitch(n);
    // Rows of block b, from its highest: i = n - 1 - RB b - s, s < RB. Each row
    // belongs to kProducers / RB warps, eight loads of each lane in flight.
    auto produce = [&](int b) {
        constexpr int kStride = 32 * (kProducers / RB);
        const int s = (warp - 1) % RB, i = n - 1 - RB * b - s;
        const int len = n - 1 - i;
        if (i >= 0 && len >= 16) {
            const double* col = f + (size_t)i * ldf + i + 1;
            const double* xi = x + i + 1;
            double* out = P + ((size_t)(b & 1) * RB + s) * pitch;
            const int n16 = len & ~15, n4 = len & ~3, full = n16 - 16, entries = 16 * list_length(len) + 4;
            // Entry e's position, or -1 for a zero.
            auto position = [&](int e) {
                if (e < full) return e + 16;
                if (e >= entries - 4) return n4 + (e - entries + 4) < len ? n4 + (e - entries + 4) : -1;
                const int u = (e - full) >> 4, l = e & 15, m = n16 + 4 * u + l;
                return l < 4 && m < n4 ? m : -1;
            };
            for (int e0 = 32 * ((warp - 1) / RB) + lane; e0 < entries; e0 += 8 * kStride) {
                double v[8];
                int m[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    m[u] = e0 + u * kStride < entries ? position(e0 + u * kStride) : -1;
                    v[u] = m[u] >= 0 ? col[m[u]] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (e0 + u * kStride < entries) out[e0 + u * kStride] = m[u] >= 0 ? mul_rn(v[u], xi[m[u]]) : 0.0;
            }
        }
        for (int e = threadIdx.x - 32; e < RB * 16; e += kThreads - 32) {
            const int s = e >> 4, m = e & 15, i = n - 1 - RB * b - s;
            head[b & 1][s][m] = i >= 0 && i + 1 + m < n ? f[(size_t)i * ldf + i + 1 + m] : 0.0;
            if (DIV && m == 0) diag[(b & 1) * RB + s] = i >= 0 ? f[(size_t)i * ldf + i] : 1.0;
        }
    };
    if (warp > 0) produce(0);
    __syncthreads();
    double xl = 0.0;  // lane L: x[i + 1 + L] of the row to come (zeros past n)
    for (int b = 0; b < blocks; ++b) {
        if (warp > 0) {
            if (b + 1 < blocks) produce(b + 1);
        } else {
#pragma unroll 1
            for (int s = 0; s < RB; ++s) {
                const int i = n - 1 - RB * b - s;
                if (i < 0) break;
                const int len = n - 1 - i;
                double* p = P + ((size_t)(b & 1) * RB + s) * pitch;
                const double rhs = x[i];
                const double p0 = mul_rn(head[b & 1][s][L], xl);
                double total;
                if (len >= 16) {
                    const int count = list_length(len);
                    const double* tail = p + 16 * count;
                    const double t0 = tail[0], t1 = tail[1], t2 = tail[2];
                    total = netdot_combine(chain<16, true>(add_rn(0.0, p0), p + L, count), L, lane & 16);
                    total = add_rn(add_rn(add_rn(total, t0), t1), t2);
                } else {
                    const int n4 = len & ~3;
                    if (lane < 16 && L < len) p[L] = p0;
                    __syncwarp();
                    total = 0.0;
                    if (len >= 4) {
                        double acc = 0.0;
                        if (L < 4)
                            for (int m = L; m < n4; m += 4) acc = add_rn(acc, p[m]);
                        __syncwarp();
                        total = netdot_combine(acc, L, lane & 16);
                    }
                    for (int m = n4; m < len; ++m) total = add_rn(total, p[m]);
                }
                double v = sub_rn(rhs, total);
                if (DIV) v = __ddiv_rn(v, diag[(b & 1) * RB + s]);
                if (lane == 0) x[i] = v;
                const double up = __shfl_up_sync(0xffffffffu, xl, 1, 16);
                xl = L == 0 ? v : up;
            }
        }
        __syncthreads();
    }
}

template <int RB>
__global__ void __launch_bounds__(kThreads) left_real_kernel(LeftSolve s, int forward, int backward) {
    extern __shared__ __align__(16) double left_smem[];
    __shared__ ForwardShared S;
    __shared__ double s_head[2][RB][16];
    __shared__ double s_diag[2 * RB];
    const int n = s.n;
    double* x = left_smem;
    double* P = x + ((n + 1) & ~1);
    double* xg = s.x + (size_t)blockIdx.x * s.ldx;
    for (int i = threadIdx.x; i < n; i += kThreads) x[i] = xg[i];
    __syncthreads();
    if (forward) forward_real(s.f, s.ldf, x, n, S);
    if (backward == (int)LowerKind::kUnit) backward_real<false, RB>(s.f, s.ldf, x, n, P, s_head, s_diag);
    else if (backward == (int)LowerKind::kDivide) backward_real<true, RB>(s.f, s.ldf, x, n, P, s_head, s_diag);
    for (int i = threadIdx.x; i < n; i += kThreads) xg[s.perm ? s.perm[i] : i] = x[i];
}

// ---- complex, L^H backward -----------------------------------------------------

// kCRows rows per phase, one column per CTA: chain lane 0 carries the real sum,
// lane 1 the imaginary one. P[buf][slot][m]: row i's product conj(f_ki) x[k] of
// position m = k - i - 1; the chain warp itself fills the positions whose x the
// phase before last did not know. A row's list, from its slot's own position q
// on, is filled with zeros to a multiple of eight.
constexpr int kCRows = 4;
__host__ __device__ inline size_t cplx_pitch(int n) { return (size_t)n + 8; }

__global__ void __launch_bounds__(kThreads) left_cplx_kernel(LeftSolve s) {
    extern __shared__ __align__(16) double left_smem[];
    __shared__ double2 s_in[2][kCRows][2 * kCRows];  // f[i + 1 + m, i] of a phase's rows, m < 8
    const int n = s.n, ldf = s.ldf;
    const double2* __restrict__ f = reinterpret_cast<const double2*>(s.f);
    double2* x = reinterpret_cast<double2*>(left_smem);  // [n]
    double2* P = x + n;                                  // [2][kCRows][pitch]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = lane & 1;
    double2* xg = reinterpret_cast<double2*>(s.x) + (size_t)blockIdx.x * s.ldx;
    for (int i = threadIdx.x; i < n; i += kThreads) x[i] = xg[i];
    __syncthreads();
    const int blocks = (n + kCRows - 1) / kCRows;
    auto row_of = [&](int b, int q) { return n - 1 - kCRows * b - q; };
    auto slot = [&](int b, int q) { return P + ((size_t)(b & 1) * kCRows + q) * cplx_pitch(n); };
    // conj(f) x in .NET's product order
    auto product = [](double2 fk, double2 xk) {
        const double ni = -fk.y;
        return make_double2(sub_rn(mul_rn(fk.x, xk.x), mul_rn(ni, xk.y)), add_rn(mul_rn(ni, xk.x), mul_rn(fk.x, xk.y)));
    };
    // Products of block b with the x solved before block b - 1: position m of
    // its row q is k = i + 1 + m; the first kCRows + q positions are later. Two
    // warps per row, four loads of each lane in flight.
    auto produce = [&](int b) {
        constexpr int kStride = 32 * (kProducers / kCRows);
        const int q = (warp - 1) % kCRows, i = row_of(b, q);
        if (i >= 0) {
            const int len = n - 1 - i, end = len > q ? q + ((len - q + 7) & ~7) : 0;  // zeros from len on
            const double2* col = f + (size_t)i * ldf + i + 1;
            for (int m0 = kCRows + q + 32 * ((warp - 1) / kCRows) + lane; m0 < end; m0 += 4 * kStride) {
                double2 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = m0 + u * kStride < len ? col[m0 + u * kStride] : make_double2(0.0, 0.0);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int m = m0 + u * kStride;
                    if (m < end) slot(b, q)[m] = m < len ? product(v[u], x[i + 1 + m]) : make_double2(0.0, 0.0);
                }
            }
        }
        for (int e = threadIdx.x - 32; e < kCRows * 2 * kCRows; e += kThreads - 32) {
            const int r = e / (2 * kCRows), m = e % (2 * kCRows), k = row_of(b, r);
            s_in[b & 1][r][m] = k >= 0 && k + 1 + m < n ? f[(size_t)k * ldf + k + 1 + m] : make_double2(0.0, 0.0);
        }
    };
    if (warp > 0) produce(0);
    __syncthreads();
    for (int b = 0; b < blocks; ++b) {
        if (warp > 0) {
            if (b + 1 < blocks) produce(b + 1);
        } else {
            // Block b - 1's x are known now: positions q .. q + kCRows - 1 of row q.
            if (lane < kCRows * kCRows) {
                const int q = lane / kCRows, m = q + lane % kCRows, i = row_of(b, q);
                if (i >= 0) slot(b, q)[m] = i + 1 + m < n ? product(s_in[b & 1][q][m], x[i + 1 + m]) : make_double2(0.0, 0.0);
            }
            __syncwarp();
            double2 own[kCRows];  // the block's x so far
#pragma unroll
            for (int q = 0; q < kCRows; ++q) {
                const int i = row_of(b, q);
                if (i < 0) break;
                const int len = n - 1 - i;
                const double* p = reinterpret_cast<const double*>(slot(b, q)) + part;
                const double2 xi = x[i];
                double sum = part ? xi.y : xi.x;
                // The block's own rows, newest first (position m = 0 is row i + 1).
#pragma unroll
                for (int m = 0; m < q; ++m) {
                    const double2 pr = product(s_in[b & 1][q][m], own[q - 1 - m]);
                    sum = sub_rn(sum, part ? pr.y : pr.x);
                }
                if (len > q) sum = chain<2, false>(sum, p + 2 * q, (len - q + 7) & ~7);
                const double other = __shfl_xor_sync(0xffffffffu, sum, 1);
                own[q] = part ? make_double2(other, sum) : make_double2(sum, other);
                if (lane == 0) x[i] = own[q];
                __syncwarp();
            }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < n; i += kThreads) xg[s.perm ? s.perm[i] : i] = x[i];
}

size_t real_smem(int n, int rb) { return sizeof(double) * (round_up(n, 2) + list_pitch(n) * 2 * rb); }
size_t cplx_smem(int n) { return sizeof(double2) * ((size_t)n + cplx_pitch(n) * 2 * kCRows); }
// The kernels' static shared memory comes out of the same 227 KB.
constexpr size_t kRealStatic = sizeof(ForwardShared) + sizeof(double) * (2 * 8 * 16 + 2 * 8);

template <class K>
void allow_smem(K kernel, std::atomic<bool>* done, int device, size_t bytes) {
    if (done[device].load(std::memory_order_acquire)) return;
    TNS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[device].store(true, std::memory_order_release);
}

}  // namespace

bool left_solve_takes(const Context& ctx, bool cplx, int n, int nrhs) {
    size_t smem = cplx ? cplx_smem(n) : real_smem(n, 8) + kRealStatic;
    if (!cplx && smem > kMaxSmem) smem = real_smem(n, 4) + kRealStatic;
    if (!cplx && smem > kMaxSmem) smem = real_smem(n, 2) + kRealStatic;
    if (smem > kMaxSmem) return false;
    // Each SM works on its right-hand sides as fast alone as together (real n =
    // 256: 0.22 ms with one each, 0.36 with two, 0.49 with three), so the time
    // goes by their rounds over the SMs; that of the staged kernels by the rounds
    // of what their shared memory holds at once, a pair to a CTA. Measured over n
    // = 32 .. 2700 real and 32 .. 1250 complex with up to 10,000 right-hand sides,
    // the staged kernels' round takes as long as these of the new (ms, real:
    // n = 64, 444: 0.17 against 0.20, 592: 0.21, 0.20; n = 512, 592: 1.31, 1.41,
    // 740: 1.60, 1.44; n = 2048, 3000: 41, 67; complex n = 256, 1500: 1.30, 1.53,
    // 6000: 4.3, 3.9; n = 1024, 1500: 31.2, 32.4, 6000: 115, 110).
    auto rounds = [&](long long at_once) { return (nrhs + at_once - 1) / at_once; };
    const double ours = (double)rounds(ctx.num_sms);
    if (n > (cplx ? kStagedCplxMaxN : kStagedRealMaxN)) {
        // The unstaged kernels, whose time hardly depends on their number (real n =
        // 4096, 16 right-hand sides: 11 against 184 ms, 2000: 134, 195, 3000: 199,
        // 202; complex n = 1400, 3000: 108, 134).
        return ours <= (cplx ? 25 : 20);
    }
    const long long ctas = std::clamp<long long>(kMaxSmem / staged_left_smem(cplx, n), 1, 32);
    const double per_round = cplx ? std::min(30.0, n < 900 ? 2048.0 / n : 1.85) : n > 64 ? 4.0 : 3.0;
    return ours <= per_round * (double)rounds(2 * ctas * ctx.num_sms);
}

namespace {
template <int RB>
bool launch_real(Context& ctx, bool forward, LowerKind backward, const LeftSolve& s) {
    const size_t room = kMaxSmem - kRealStatic, smem = real_smem(s.n, RB);
    if (smem > room) return false;
    static std::atomic<bool> done[64];
    allow_smem(left_real_kernel<RB>, done, ctx.device, room);
    left_real_kernel<RB><<<s.nrhs, kThreads, smem, ctx.stream>>>(s, forward, (int)backward);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
    return true;
}
}  // namespace

void left_solve_real(Context& ctx, bool forward, LowerKind backward, const LeftSolve& s) {
    if (s.n == 0 || s.nrhs == 0) return;
    if (launch_real<8>(ctx, forward, backward, s) || launch_real<4>(ctx, forward, backward, s) ||
        launch_real<2>(ctx, forward, backward, s))
        return;
    fail(TNS_E_ARGUMENT, "internal: left-looking solve too large for its kernel");
}

void left_solve_cplx(Context& ctx, const LeftSolve& s) {
    if (s.n == 0 || s.nrhs == 0) return;
    static std::atomic<bool> done[64];
    allow_smem(left_cplx_kernel, done, ctx.device, kMaxSmem);
    left_cplx_kernel<<<s.nrhs, kThreads, cplx_smem(s.n), ctx.stream>>>(s);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
}

}  // namespace tns
