// exp(tA)B by Al-Mohy & Higham 2011 truncated Taylor (the reference's
// MatrixExponentialAction.Dense + Run, src/Tensile/MatrixExponentialAction.cs:149-178,
// 239-320), for one matrix or a batch of independent ones.
//
// The parameter selection runs on the host in the reference's order (trace
// shift, ||A - mu I||_1, the sharp ||A^p||^(1/p) bounds from normest1 with
// every estimator of the batch advanced together, the (m, s) search). The
// whole Taylor recurrence -- every operator application, the scaling of the
// new term, its accumulation into F, both infinity norms and the early-exit
// test -- then runs in ONE cooperative launch: taylor_kernel.
//
// taylor_kernel. Each matrix is worked on by a group of CTAs ("lanes"); the
// rows of A, F and the work panels are split among them. One application of
// A to the n x c work panel X is, per CTA, the product of its rows of A with
// all of X, summed in k order with the reference's rounding (PanelProduct.Apply's
// axpy order, a product and a sum per term; the complex operator's four real
// sums then (pr - qi, pi + qr), LinearOperators.cs:262-282). The reference skips
// a term whose x is zero; forming it instead adds +-0 to a sum that is never
// -0, which changes nothing as long as A is finite, so the skip is kept (as a
// compare and a select) only in launches with a non-finite operator. The
// epilogue scales the sums by t/(s(j+1)) into the next work panel, adds them
// into F and forms both row sums of moduli in column order (InfinityNorm). The
// group then meets at a barrier that also exchanges the two norms, and every
// CTA takes the same exit decision: c1 + c2 <= u ||F||_inf ends the inner loop
// on the device, with no host round trip. The panels alternate between two
// buffers, so no CTA overwrites a panel another is still reading.
//
// What bounds it: FP64 issue (a product and a sum per term, not fused: 8
// instructions per complex term, 17.6 cycles of a partition per 4 rows x 8
// columns) and, per application, the epilogue's and the barrier's latencies.
// A staging thread keeps a ring of tiles filled by TMA (a box of A, whose
// first tiles of the next application are fetched while this one ends, and a
// piece of the row-major X); the multiplying warps hold several rows each,
// with loads, products and sums of three successive k's in flight. On 24
// complex matrices (64..1024, 8 columns, 22538 applications) the launch takes
// 64 ms of which the FP64 instructions alone would take 32; per-thread
// staging with one row and column per thread, a barrier per tile and a branch
// per column took 120.
//
// Groups and the barrier. A host-side list schedule gives each matrix a width
// (CTAs) and places it, longest first, on the lanes that free up earliest;
// each CTA then works through its list of (matrix, rank) in the order of the
// schedule's start times, which is one total order for every lane, so no
// group can wait on a lane that waits on it. A group of one CTA synchronises
// with __syncthreads; a wider group through slots in global memory, with a
// bounded spin: a wait gives up after 2 s in which no barrier anywhere in the
// launch advanced, records a device error and returns, and the host reports
// TNS_E_TIMEOUT.

#include "batch.cuh"
#include "device_util.cuh"
#include "net_compat.h"
#include "tns_internal.h"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <limits>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

namespace tns {

namespace {

constexpr int kMultiplyT = 256;           // threads of the multiplying warps: two groups of four
constexpr int kThreadsT = kMultiplyT + 32;  // and the staging warp

// The thread layout and the inner loop's form, per launch: SLOTS column slots
// per row, CPT columns per slot (c + SLOTS q), UNIT rows per step of a group
// of multiplying warps, up to UMAX steps (the first group takes the odd one)
// and so up to ROWS rows per chunk of a CTA's row range.
// SKIP keeps the reference's skip of a zero x term explicitly (a compare and
// a select per term). Without it the term is always formed: that adds +-0 to
// a sum that is never -0, the same bits whenever A is finite; the host takes
// that form only when every ||A - mu I||_1 of the launch is finite (0 * inf
// would otherwise differ from a skip).
template <int SLOTS_, int CPT_, int UMAX_, bool SKIP_>
struct Shape {
    static constexpr int SLOTS = SLOTS_, CPT = CPT_, UMAX = UMAX_;
    static constexpr int COLS = SLOTS * CPT, UNIT = 128 / SLOTS, ROWS = UNIT * UMAX;
    static constexpr bool SKIP = SKIP_;
};
// k per staged tile of a chunk's rows and the panel's columns: long tiles where they are few (a
// tile costs its warps some 200 cycles besides the products). Chunks stop at
// 112 rows, of which three stages of 32 fit; 128 rows in stages of 16 took
// 207 to 222 cycles a k, 112 rows 150 (8 columns, complex).
__host__ __device__ constexpr int tile_k(int rows, int cols) {
    return rows + cols <= 24 ? 128 : rows + cols <= 40 ? 64 : 32;
}
constexpr int kStagesMax = 8;              // ring depth, as far as kSmemT holds it
constexpr size_t kSmemT = 222 * 1024;      // dynamic shared memory of a CTA
constexpr double kU = 1.1102230246251565e-16;
constexpr int kDevTimeoutGroup = 4;  // DeviceError: a group barrier of the Taylor kernel gave up

struct TaylorDesc {
    const double* b;   // B, ld ldb
    double* f;         // the result F, ld ldp
    double* w0;        // work panels, row-major, COLS wide
    double* w1;
    const double* coeff;        // m coefficients t / (s (j + 1))
    unsigned long long* slots;  // [3][width][2] norms, kEmpty until published
    int* out;                   // [applications, early exits]
    int n, ldb, ldp;
    int m, s, width, chunk, rows_per;  // rows_per: rows per CTA and per chunk of them, multiples of the launch's UNIT
    double eta_re, eta_im;
    int eta_one;
};

struct TaylorPlan {
    int matrix, rank;
};

struct TaylorLaunch {
    const TaylorDesc* descs;
    const TaylorPlan* plan;
    const CUtensorMap* maps;  // of each shifted matrix, boxes of a chunk's rows by tile_k columns
    const int* plan_off;  // gridDim.x + 1 offsets into plan
    int ncols;
    int* err;
    unsigned long long* progress;  // every barrier arrival in the launch
};

// Orders this thread's plain accesses to global memory with bulk copies of it.
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// Two words, each read whole.
__device__ __forceinline__ ulonglong2 ld_acquire2(const unsigned long long* p) {
    ulonglong2 v;
    asm volatile("ld.acquire.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Largest of non-negative values with Math.Max's NaN rule (any NaN wins):
// their bits order as the values do, a quiet NaN above infinity.
struct NormAcc {
    unsigned long long bits = 0;
    __device__ void add(double x) { join(isnan(x) ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(x)); }
    __device__ void join(unsigned long long b) { bits = b > bits ? b : bits; }
    // Over the warp: the high words' largest, then the low words' among its.
    __device__ void fold() {
        const unsigned hi = (unsigned)(bits >> 32), top = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lo = hi == top ? (unsigned)bits : 0u;
        bits = ((unsigned long long)top << 32) | __reduce_max_sync(0xffffffffu, lo);
    }
};
constexpr unsigned long long kEmpty = ~0ull;  // a slot not yet published (no norm has these bits)

struct NormShared {
    unsigned long long warp[2][kThreadsT / 32];
    double norm[2];
    int ok;
};

// Join the group's published words of this lane's ranks, all of them asked
// for at once until each is there. False when the wait gave up.
__device__ bool await_slots(const unsigned long long* slots, int width, const TaylorLaunch& L, NormAcc& r0, NormAcc& r1) {
    unsigned long long start = 0, beat = 0;
    for (unsigned it = 0;; ++it) {
        bool all = true;
        for (int r = threadIdx.x; r < width; r += 32) {
            const ulonglong2 v = ld_acquire2(slots + 2 * r);
            if (v.x != kEmpty) r0.join(v.x);
            if (v.y != kEmpty) r1.join(v.y);
            all = all && v.x != kEmpty && v.y != kEmpty;
        }
        if (all) return true;
        if (it > 64) __nanosleep(64);
        if ((it & 127u) == 0) {
            if (*reinterpret_cast<volatile int*>(L.err) != 0) return false;
            const unsigned long long now = global_timer_ns(), b2 = ld_relaxed(L.progress);
            if (it == 0 || b2 != beat) {
                beat = b2;
                start = now;
            } else if (now - start > kWaitTimeoutNs) {
                atomicCAS(L.err, 0, kDevTimeoutGroup);
                return false;
            }
        }
    }
}

// The group's barrier and its two norms (sh.norm, every thread): each CTA
// publishes its own two and reads everyone's, so that arriving and giving the
// value are one store, and waiting and reading it one load (4600 cycles for a
// group of 4 with a counter, a fence on each side and the values read after
// it; 2700 to 3500 so).
// Slots rotate over three phases. A CTA empties its slot of phase p + 2 after
// it has seen all of phase p, when everyone has read phase p - 1, the slot's
// last use; and it publishes p + 1, which everyone awaits before p + 2, after
// that. False if a wait gave up here or on the ring of tiles.
__device__ bool group_norms(const TaylorDesc& d, int rank, unsigned& phase, const TaylorLaunch& L, NormAcc a0,
                            NormAcc a1, NormShared& sh, const int* s_dead) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    fence_async_global();  // this thread's part of the work panel, before the group's copies of it
    a0.fold();
    a1.fold();
    if (lane == 0) {
        sh.warp[0][warp] = a0.bits;
        sh.warp[1][warp] = a1.bits;
    }
    __syncthreads();
    if (warp == 0) {
        NormAcc r0, r1;
        if (lane < kThreadsT / 32) {
            r0.bits = sh.warp[0][lane];
            r1.bits = sh.warp[1][lane];
        }
        r0.fold();
        r1.fold();
        bool ok = true;
        if (d.width > 1) {
            unsigned long long* slots = d.slots + (size_t)phase * d.width * 2;
            if (lane == 0) {
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                st_relaxed(slots + 2 * rank, r0.bits);
                st_relaxed(slots + 2 * rank + 1, r1.bits);
            }
            ok = await_slots(slots, d.width, L, r0, r1);
            __syncwarp();
            r0.fold();
            r1.fold();
            ok = __all_sync(0xffffffffu, ok);
            phase = phase == 2 ? 0 : phase + 1;
            if (lane == 0) atomicAdd(L.progress, 1ull);  // the launch is alive
            if (lane < 2) st_relaxed(d.slots + (size_t)(phase == 2 ? 0 : phase + 1) * d.width * 2 + 2 * rank + lane, kEmpty);
        }
        if (lane == 0) {
            sh.norm[0] = __longlong_as_double((long long)r0.bits);
            sh.norm[1] = __longlong_as_double((long long)r1.bits);
            sh.ok = ok;
        }
    } else if (d.width > 1) {
        phase = phase == 2 ? 0 : phase + 1;
    }
    __syncthreads();
    return sh.ok && !*s_dead;
}

template <bool CPLX>
__device__ __forceinline__ double modulus(double re, double im) {
    if constexpr (CPLX) return cabs_net(re, im);
    else return fabs(re);
}

// Row sums of moduli over the columns in column order (InfinityNorm,
// ComplexKernels.cs:164-180 / Norms.cs:50-66): the 8 lanes of a row hold its
// columns c + SLOTS q; every lane ends with its row's sum.
template <class S>
__device__ __forceinline__ double row_sum(const double (&v)[S::CPT], int ncols) {
    const int base = threadIdx.x & (32 - S::SLOTS);  // first lane of this row in the warp
    double sum = 0.0;
#pragma unroll
    for (int q = 0; q < S::CPT; ++q)
#pragma unroll
        for (int c = 0; c < S::SLOTS; ++c) {
            const double x = __shfl_sync(0xffffffffu, v[q], base + c);
            if (q * S::SLOTS + c < ncols) sum = add_rn(sum, x);
        }
    return sum;
}

template <bool CPLX, class S>
struct Tiles {
    static constexpr int ES = CPLX ? 2 : 1;              // doubles per element
    static constexpr int Y_DOUBLES = S::ROWS * S::COLS * ES;  // of the products, and of F
    // One stage for chunks of up to `units` steps of rows, and how many fit.
    static __host__ __device__ constexpr int stage_doubles(int units) {
        return tile_k(S::UNIT * units, S::COLS) * (S::UNIT * units + S::COLS) * ES;
    }
    static __device__ __forceinline__ int stages(int units) {
        return min(kStagesMax, (int)((kSmemT / sizeof(double) - 2 * Y_DOUBLES) / stage_doubles(units)));
    }
    static_assert(stage_doubles(S::UMAX) * 3 + 2 * Y_DOUBLES <= (int)(kSmemT / sizeof(double)), "three stages");
    static_assert(S::ROWS * ES <= 256, "the rows of a tensor-map box");
    static_assert(S::UNIT * S::COLS * ES * 8 % 128 == 0, "TMA destinations at multiples of 128 bytes");
};

// A position in the ring of staged tiles: the slot and the parity of its lap.
struct Ring {
    int slot = 0;
    unsigned lap = 0;
    __device__ void next(int stages) {
        if (++slot == stages) {
            slot = 0;
            lap ^= 1;
        }
    }
};

struct RingBars {
    uint64_t full[kStagesMax], empty[kStagesMax];
    int dead;  // a wait on the ring gave up
};

// The staging warp's side, one thread of it: k tile [k0, k0 + kt) of the
// CTA's rows r0... of A into a slot of the ring, one box of `units` steps of
// rows (those past the matrix come as zeros), and the same rows of the work
// panel. (Copies of single columns of the tile kept the staging warp busy for
// 1900 cycles a tile, and per-thread copies four warps for 2900, against 900
// to multiply 16 rows of it.)
template <bool CPLX, class S>
struct Stager {
    using T = Tiles<CPLX, S>;
    const TaylorDesc& d;
    const CUtensorMap* map;
    double* smem;
    RingBars& bars;
    int* err;
    int units, kt, stages, stage_doubles;
    Ring a, x;  // the next tile of A and of X

    __device__ __forceinline__ bool put_a(int r0, int k0) {
        if (!mbar_wait_bounded(&bars.empty[a.slot], a.lap ^ 1, err, kDevTimeoutEmpty)) {
            bars.dead = 1;
            return false;
        }
        mbar_arrive_expect_tx(&bars.full[a.slot], kt * S::UNIT * units * T::ES * 8);
        tma_load_2d(smem + (size_t)a.slot * stage_doubles, map, r0 * T::ES, k0, &bars.full[a.slot]);
        a.next(stages);
        return true;
    }
    __device__ __forceinline__ void put_x(const double* w, int k0) {
        const uint32_t bytes = min(kt, d.n - k0) * S::COLS * T::ES * 8;
        mbar_arrive_expect_tx(&bars.full[x.slot], bytes);
        bulk_copy_g2s(smem + (size_t)x.slot * stage_doubles + kt * S::UNIT * units * T::ES,
                      w + (size_t)k0 * S::COLS * T::ES, bytes, &bars.full[x.slot]);
        x.next(stages);
    }
    // Tiles of A without their X: take their copies in, so that none is under
    // way when the slots are given up; likewise, after a wait that gave up,
    // the last tile of every slot.
    __device__ void drain() {
        while (x.slot != a.slot || x.lap != a.lap) {
            mbar_arrive(&bars.full[x.slot]);
            x.next(stages);
        }
        for (int s = 0; s < stages; ++s)
            mbar_wait_bounded(&bars.full[s], s < a.slot ? a.lap : a.lap ^ 1, err, kDevTimeoutDrain);
    }
};

// Steps of rows of the first group of four multiplying warps: all of up to
// three, half from four on. One warp per partition with two rows a thread
// takes 41 cycles a k, two with one each 54; with four and two 76 and 75, and
// beyond that two warps hide each other's latencies (8 columns, complex).
__host__ __device__ constexpr int first_steps(int units) { return units <= 3 ? units : (units + 1) / 2; }

// The multiplying warps' side: Y := (rows of the chunk of A) X over all k
// tiles, in k order, into sY (row-major, COLS wide). Thread (row, column) of
// a group holds rows row + UNIT (base + q): a warp reads RT + CPT operands
// for 8 RT CPT (complex) FP64 instructions. The operands of k + 2 are loaded
// and the products of k + 1 formed while those of k are added, across the
// tiles' ends. Columns past ncols repeat the last.
template <bool CPLX, class S, int RT>
__device__ __forceinline__ void multiply_chunk(double* smem, RingBars& bars, Ring& ring, int stages, int stage_doubles,
                                               int kt, int pitch, int base, int n, int ncols, double* sY, int* err) {
    using T = Tiles<CPLX, S>;
    constexpr int CPT = S::CPT;
    using Elem = std::conditional_t<CPLX, double2, double>;
    // Bit 1 of the lane counts rows and bit 0 columns, so that lanes a bit
    // apart read the same operand: a 16-byte read of a warp then takes two
    // passes instead of four, of A and of X both.
    const int lane = threadIdx.x & 31, c = (lane & 1) | ((lane >> 1) & (S::SLOTS - 2));
    const int rr = base * S::UNIT + (threadIdx.x % 128 >> 5) * (32 / S::SLOTS) +
                   (((lane >> 1) & 1) | (lane / (2 * S::SLOTS) * 2));
    double acc[RT][CPT][CPLX ? 4 : 1];
#pragma unroll
    for (int q = 0; q < RT; ++q)
#pragma unroll
        for (int p = 0; p < CPT; ++p)
#pragma unroll
            for (int z = 0; z < (CPLX ? 4 : 1); ++z) acc[q][p][z] = 0.0;
    int xoff[CPT];
#pragma unroll
    for (int p = 0; p < CPT; ++p) xoff[p] = min(c + p * S::SLOTS, ncols - 1);
    bool alive = true;
    const Elem *sA, *sX;
    Elem av[2][RT], xv[2][CPT];
    // The next tile. After a wait that gave up the sums are of no use, and the
    // CTA returns at its next barrier.
    auto take = [&] {
        if (alive && !mbar_wait_bounded(&bars.full[ring.slot], ring.lap, err, kDevTimeoutFull)) {
            alive = false;
            bars.dead = 1;
        }
        sA = reinterpret_cast<const Elem*>(smem + (size_t)ring.slot * stage_doubles) + rr;
        sX = reinterpret_cast<const Elem*>(smem + (size_t)ring.slot * stage_doubles) + kt * pitch;
    };
    auto load = [&](int b, int k) {
#pragma unroll
        for (int q = 0; q < RT; ++q) av[b][q] = sA[k * pitch + q * S::UNIT];
#pragma unroll
        for (int p = 0; p < CPT; ++p) xv[b][p] = sX[k * S::COLS + xoff[p]];
    };
    double pr[2][RT][CPT][CPLX ? 4 : 1];
    auto multiply = [&](int b) {
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int p = 0; p < CPT; ++p) {
                if constexpr (CPLX) {
                    const double2 a = av[b][q], x = xv[b][p];
                    const bool nr = !S::SKIP || x.x != 0.0, ni = !S::SKIP || x.y != 0.0;
                    pr[b][q][p][0] = nr ? mul_rn(x.x, a.x) : 0.0;  // pr
                    pr[b][q][p][1] = ni ? mul_rn(x.y, a.x) : 0.0;  // pi
                    pr[b][q][p][2] = nr ? mul_rn(x.x, a.y) : 0.0;  // qr
                    pr[b][q][p][3] = ni ? mul_rn(x.y, a.y) : 0.0;  // qi
                } else {
                    const double a = av[b][q], x = xv[b][p];
                    pr[b][q][p][0] = !S::SKIP || x != 0.0 ? mul_rn(x, a) : 0.0;
                }
            }
    };
    auto add = [&](int b) {
#pragma unroll
        for (int q = 0; q < RT; ++q)
#pragma unroll
            for (int p = 0; p < CPT; ++p)
#pragma unroll
                for (int z = 0; z < (CPLX ? 4 : 1); ++z) acc[q][p][z] = add_rn(acc[q][p][z], pr[b][q][p][z]);
    };
    take();
    load(0, 0);
    load(1, 1);
    multiply(0);
    for (int k0 = 0; k0 < n; k0 += kt) {
        const int klen = min(kt, n - k0);
        const bool more = k0 + kt < n;
        uint64_t* done = &bars.empty[ring.slot];
        ring.next(stages);
        // (loads past the last k: whatever the slot holds there, not used)
        int kk = 0;
        for (; kk + 4 <= klen - (more ? 4 : 0); kk += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                load(u & 1, kk + u + 2);
                multiply((u + 1) & 1);
                add(u & 1);
            }
        }
        if (more) {
            // The last four, with the first operands of the next tile.
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (u == 2) take();
                load(u & 1, u < 2 ? kk + u + 2 : u - 2);
                multiply((u + 1) & 1);
                add(u & 1);
            }
        } else {
#pragma unroll
            for (int u = 0; u < 3; ++u)
                if (kk + u < klen) {
                    load(u & 1, kk + u + 2);
                    multiply((u + 1) & 1);
                    add(u & 1);
                }
        }
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(done);
    }
#pragma unroll
    for (int q = 0; q < RT; ++q)
#pragma unroll
        for (int p = 0; p < CPT; ++p) {
            double* y = sY + ((q * S::UNIT + rr) * S::COLS + c + p * S::SLOTS) * T::ES;
            if constexpr (CPLX) {
                // the reference's four real sums combine as (pr - qi, pi + qr)
                *reinterpret_cast<double2*>(y) = make_double2(sub_rn(acc[q][p][0], acc[q][p][3]), add_rn(acc[q][p][1], acc[q][p][2]));
            } else {
                y[0] = acc[q][p][0];
            }
        }
}

template <bool CPLX, class S, int RT = (S::UMAX > 6 ? (S::UMAX + 1) / 2 : 3)>
__device__ __forceinline__ void multiply_dispatch(int rt, double* smem, RingBars& bars, Ring& ring, int stages,
                                                  int stage_doubles, int kt, int pitch, int base, int n, int ncols, double* sY,
                                                  int* err) {
    if constexpr (RT == 0) {
        // The second group of a chunk of one step: frees the tiles unread.
        for (int k0 = 0; k0 < n; k0 += kt) {
            if (!mbar_wait_bounded(&bars.full[ring.slot], ring.lap, err, kDevTimeoutFull)) bars.dead = 1;
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbar_arrive(&bars.empty[ring.slot]);
            ring.next(stages);
        }
    } else {
        if (rt == RT)
            return multiply_chunk<CPLX, S, RT>(smem, bars, ring, stages, stage_doubles, kt, pitch, base, n, ncols, sY, err);
        multiply_dispatch<CPLX, S, RT - 1>(rt, smem, bars, ring, stages, stage_doubles, kt, pitch, base, n, ncols, sY, err);
    }
}

template <bool CPLX, class S>
__global__ void __launch_bounds__(kThreadsT, 1) taylor_kernel(const __grid_constant__ TaylorLaunch L) {
    using T = Tiles<CPLX, S>;
    constexpr int CPT = S::CPT, ES = T::ES;
    constexpr int RP = kMultiplyT / S::SLOTS;  // rows of one pass of the element-wise parts
    extern __shared__ __align__(128) double smem[];
    __shared__ RingBars bars;
    __shared__ NormShared sh;
    double* const sY = smem + kSmemT / sizeof(double) - 2 * T::Y_DOUBLES;
    double* const sF = sY + T::Y_DOUBLES;
    const int ncols = L.ncols;
    const bool multiplying = threadIdx.x < kMultiplyT;
    const int rr = multiplying ? threadIdx.x / S::SLOTS : 1 << 28, cs = threadIdx.x % S::SLOTS;
    const bool staging = threadIdx.x == kMultiplyT;
    if (threadIdx.x == 0) bars.dead = 0;
    for (int e = L.plan_off[blockIdx.x]; e < L.plan_off[blockIdx.x + 1]; ++e) {
        const TaylorPlan pl = L.plan[e];
        const TaylorDesc d = L.descs[pl.matrix];
        const int rank = pl.rank;
        const int rbeg = rank * d.rows_per, rend = min(d.n, rbeg + d.rows_per);
        const int R = d.chunk, units = R / S::UNIT, kt = tile_k(R, S::COLS);  // of the staged boxes
        const int ktiles = (d.n + kt - 1) / kt;
        const int stage_doubles = T::stage_doubles(units), stages = T::stages(units);
        unsigned phase = 0;
        if (threadIdx.x == 0) {
            for (int i = 0; i < stages; ++i) {
                mbar_init(&bars.full[i], 2);
                mbar_init(&bars.empty[i], kMultiplyT / 32);
            }
            mbar_fence_init();
        }
        __syncthreads();
        // A does not change: its first tiles of the next product are copied
        // ahead of the barrier that X waits for.
        Ring ring;  // the multiplying warps' next tile
        Stager<CPLX, S> st{d, L.maps + pl.matrix, smem, bars, L.err, units, kt, stages, stage_doubles};
        const int ahead = min(stages, ktiles);
        // F stays in shared memory to the end where the CTA's rows are one chunk.
        const bool f_local = rend - rbeg <= R;
        auto f_at = [&](int i, int col) {
            return f_local ? sF + ((i - rbeg) * S::COLS + col) * ES : d.f + ((size_t)col * d.ldp + i) * ES;
        };
        if (staging) {
            tensormap_acquire(st.map);
            for (int t = 0; t < ahead && st.put_a(rbeg, t * kt); ++t) {}
        }

        // F := B, work := B, c1 = ||B||_inf (Run, :274-276, :285).
        NormAcc n0, n1;
        for (int r0 = rbeg; r0 < rend; r0 += RP) {
            const int i = r0 + rr;
            const bool row_ok = i < rend;
            double v[CPT];
#pragma unroll
            for (int q = 0; q < CPT; ++q) {
                const int col = cs + q * S::SLOTS;
                v[q] = 0.0;
                if (row_ok && col < ncols) {
                    const size_t bi = ((size_t)col * d.ldb + i) * ES;
                    double* f = f_at(i, col);
                    const size_t wi = ((size_t)i * S::COLS + col) * ES;
                    const double re = d.b[bi], im = CPLX ? d.b[bi + 1] : 0.0;
                    f[0] = re;
                    d.w0[wi] = re;
                    if (CPLX) {
                        f[1] = im;
                        d.w0[wi + 1] = im;
                    }
                    v[q] = modulus<CPLX>(re, im);
                }
            }
            const double rs = row_sum<S>(v, ncols);
            if (row_ok) n0.add(rs);
        }
        if (!group_norms(d, rank, phase, L, n0, n1, sh, &bars.dead)) {
            if (staging) st.drain();
            return;
        }
        double c1 = sh.norm[0];

        int applications = 0, early = 0;
        double* win = d.w0;
        double* wout = d.w1;
        for (int step = 0; step < d.s; ++step) {
            for (int j = 0; j < d.m; ++j) {
                const double coeff = d.coeff[j];
                NormAcc nw, nf;
                for (int c0 = rbeg; c0 < rend; c0 += R) {
                    const int rows = min(R, rend - c0);
                    if (staging) {
                        fence_async_global();
                        bool ok = true;
                        for (int t = 0; t < ktiles && ok; ++t) {
                            if (t >= ahead) ok = st.put_a(c0, t * kt);
                            if (ok) st.put_x(win, t * kt);
                        }
                        const int next = c0 + R < rend ? c0 + R : rbeg;
                        for (int t = 0; t < ahead && ok; ++t) ok = st.put_a(next, t * kt);
                    } else if (multiplying) {
                        const int u = (rows + S::UNIT - 1) / S::UNIT, first = first_steps(u), second = threadIdx.x >> 7;
                        multiply_dispatch<CPLX, S>(second ? u - first : first, smem, bars, ring, stages, stage_doubles,
                                                   kt, units * S::UNIT, second ? first : 0, d.n, ncols, sY, L.err);
                    }
                    __syncthreads();
#pragma unroll 2
                    for (int b = 0; b < rows; b += RP) {
                        const int r = b + rr, i = c0 + r;
                        const bool row_ok = r < rows;
                        double vw[CPT], vf[CPT];
#pragma unroll
                        for (int q = 0; q < CPT; ++q) {
                            const int col = cs + q * S::SLOTS;
                            vw[q] = 0.0;
                            vf[q] = 0.0;
                            if (row_ok && col < ncols) {
                                double* f = f_at(i, col);
                                double* w = wout + ((size_t)i * S::COLS + col) * ES;
                                const double* y = sY + (r * S::COLS + col) * ES;
                                if constexpr (CPLX) {
                                    // next = A work; work := Scale(next, coefficient) (ScaleInto, :441-452)
                                    const double wr = mul_rn(y[0], coeff), wi = mul_rn(y[1], coeff);
                                    *reinterpret_cast<double2*>(w) = make_double2(wr, wi);
                                    // F += work (AddInto, :466-476)
                                    const double fr = add_rn(f[0], wr), fi = add_rn(f[1], wi);
                                    f[0] = fr;
                                    f[1] = fi;
                                    vw[q] = cabs_net(wr, wi);
                                    vf[q] = cabs_net(fr, fi);
                                } else {
                                    const double wr = mul_rn(y[0], coeff);
                                    w[0] = wr;
                                    const double fv = add_rn(f[0], wr);
                                    f[0] = fv;
                                    vw[q] = fabs(wr);
                                    vf[q] = fabs(fv);
                                }
                            }
                        }
                        const double sw = row_sum<S>(vw, ncols), sf = row_sum<S>(vf, ncols);
                        if (row_ok) {
                            nw.add(sw);
                            nf.add(sf);
                        }
                    }
                    if (c0 + R < rend) __syncthreads();  // the next chunk's products overwrite sY
                }
                if (!group_norms(d, rank, phase, L, nw, nf, sh, &bars.dead)) {
                    if (staging) st.drain();
                    return;
                }
                const double c2 = sh.norm[0], fnorm = sh.norm[1];
                ++applications;
                double* tmp = win;
                win = wout;
                wout = tmp;
                // The remaining terms cannot move F at this precision (:298-305).
                if (add_rn(c1, c2) <= mul_rn(kU, fnorm)) {
                    ++early;
                    break;
                }
                c1 = c2;
            }
            // F *= eta (ScaleInPlace, :455-464); work := F (CopyInto); c1 = ||work||_inf.
            NormAcc ne, unused;
            for (int r0 = rbeg; r0 < rend; r0 += RP) {
                const int i = r0 + rr;
                const bool row_ok = i < rend;
                double v[CPT];
#pragma unroll
                for (int q = 0; q < CPT; ++q) {
                    const int col = cs + q * S::SLOTS;
                    v[q] = 0.0;
                    if (row_ok && col < ncols) {
                        double* f = f_at(i, col);
                        double re = f[0], im = CPLX ? f[1] : 0.0;
                        if (!d.eta_one) {
                            if constexpr (CPLX) {
                                // Complex multiply (left = F, right = eta), .NET's order of terms.
                                const double nr = sub_rn(mul_rn(re, d.eta_re), mul_rn(im, d.eta_im));
                                const double ni = add_rn(mul_rn(im, d.eta_re), mul_rn(re, d.eta_im));
                                re = nr;
                                im = ni;
                            } else {
                                re = mul_rn(re, d.eta_re);
                            }
                            f[0] = re;
                            if (CPLX) f[1] = im;
                        }
                        double* w = win + ((size_t)i * S::COLS + col) * ES;
                        w[0] = re;
                        if (CPLX) w[1] = im;
                        v[q] = modulus<CPLX>(re, im);
                    }
                }
                const double rs = row_sum<S>(v, ncols);
                if (row_ok) ne.add(rs);
            }
            if (!group_norms(d, rank, phase, L, ne, unused, sh, &bars.dead)) {
                if (staging) st.drain();
                return;
            }
            c1 = sh.norm[0];
        }
        if (rank == 0 && threadIdx.x == 0) {
            d.out[0] = applications;
            d.out[1] = early;
        }
        if (f_local)
            for (int i = rbeg + rr; i < rend; i += RP)
#pragma unroll
                for (int q = 0; q < CPT; ++q) {
                    const int col = cs + q * S::SLOTS;
                    if (col < ncols)
                        for (int z = 0; z < ES; ++z) d.f[((size_t)col * d.ldp + i) * ES + z] = f_at(i, col)[z];
                }
        // The tiles of A copied ahead for a product that never came.
        if (staging) st.drain();
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 0; i < stages; ++i) {
                mbar_inval(&bars.full[i]);
                mbar_inval(&bars.empty[i]);
            }
        __syncthreads();
    }
}

// ---- host ----------------------------------------------------------------

__global__ void trace_batch_kernel(const __grid_constant__ Batch<SumDesc> b, bool cplx) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= b.count) return;
    const SumDesc& d = batch_item(b, k);
    double re = 0.0, im = 0.0;
    for (int i = 0; i < d.m; ++i) {
        if (!cplx) {
            re = add_rn(re, d.a[(size_t)i * d.ld + i]);
        } else {
            const double2 z = reinterpret_cast<const double2*>(d.a)[(size_t)i * d.ld + i];
            re = add_rn(re, z.x);
            im = add_rn(im, z.y);
        }
    }
    d.out[0] = re;
    d.out[1] = im;
}

// The trace of every matrix (Trace, :418-423; complex per part), to the host.
std::vector<double> traces(Context& ctx, const std::vector<const DMat*>& as) {
    const size_t cnt = as.size();
    DBuf out(ctx, sizeof(double) * 2 * cnt);
    std::vector<SumDesc> v;
    for (size_t k = 0; k < cnt; ++k) v.push_back(SumDesc{as[k]->p, as[k]->rows, as[k]->rows, as[k]->ld(), out.as<double>() + 2 * k});
    Batch<SumDesc> b = make_batch(ctx, v);
    trace_batch_kernel<<<(int)((cnt + 127) / 128), 128, 0, ctx.stream>>>(b, as[0]->cplx);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
    std::vector<double> h(2 * cnt);
    TNS_CUDA(cudaMemcpyAsync(h.data(), out.p, sizeof(double) * 2 * cnt, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    return h;
}

const int kEll = 2, kMaxPower = 8;

template <bool CPLX, class S>
void launch_taylor(Context& ctx, const TaylorLaunch& L, int grid) {
    TNS_CUDA(cudaFuncSetAttribute(taylor_kernel<CPLX, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemT));
    void* args[] = {const_cast<TaylorLaunch*>(&L)};
    TNS_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(taylor_kernel<CPLX, S>), dim3(grid),
                                         dim3(kThreadsT), args, kSmemT, ctx.stream));
    ctx.kernel_launches++;
}

template <bool CPLX, class S>
int resident_ctas(Context& ctx) {
    TNS_CUDA(cudaFuncSetAttribute(taylor_kernel<CPLX, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemT));
    int per_sm = 0;
    TNS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, taylor_kernel<CPLX, S>, kThreadsT, kSmemT));
    if (per_sm < 1) fail(TNS_E_DEVICE, "the Taylor kernel cannot be resident on this device");
    return per_sm * ctx.num_sms;
}

// What the host needs of a launch's Shape.
struct Layout {
    int cols, unit, rows, lanes;  // panel pitch, rows per step, rows per box at most, resident CTAs
};

// One kernel instance per (element type, layout, skip form); L null: only its
// Layout.
template <bool CPLX, class S>
Layout taylor_shape(Context& ctx, const TaylorLaunch* L, int grid) {
    if (L) launch_taylor<CPLX, S>(ctx, *L, grid);
    return Layout{S::COLS, S::UNIT, S::ROWS, L ? grid : resident_ctas<CPLX, S>(ctx)};
}

// Layouts by panel width: up to 4, 8, 16 and 32 columns.
template <bool CPLX, bool SKIP>
Layout taylor_dispatch(Context& ctx, int ncols, const TaylorLaunch* L, int grid) {
    if (ncols <= 4) return taylor_shape<CPLX, Shape<4, 1, 3, SKIP>>(ctx, L, grid);
    if (ncols <= 8) return taylor_shape<CPLX, Shape<8, 1, 7, SKIP>>(ctx, L, grid);
    if (ncols <= 16) return taylor_shape<CPLX, Shape<16, 1, 8, SKIP>>(ctx, L, grid);
    return taylor_shape<CPLX, Shape<16, 2, 4, SKIP>>(ctx, L, grid);
}

Layout taylor(Context& ctx, bool cplx, bool skip, int ncols, const TaylorLaunch* L, int grid) {
    if (cplx) return skip ? taylor_dispatch<true, true>(ctx, ncols, L, grid) : taylor_dispatch<true, false>(ctx, ncols, L, grid);
    return skip ? taylor_dispatch<false, true>(ctx, ncols, L, grid) : taylor_dispatch<false, false>(ctx, ncols, L, grid);
}

// The schedule: each matrix's width (CTAs) and rows per CTA, and the per-lane
// lists of (matrix, rank) sorted by (start time, placement order).
struct Sched {
    std::vector<int> width, rows_per;
    std::vector<int> offsets;
    std::vector<TaylorPlan> plan;
    double makespan = 0.0;
};

// A CTA's rows in the fewest chunks of up to `most` rows, evenly: a short
// last chunk costs far more per row than a full one.
int chunk_rows(int rows, int unit, int most) {
    const int units = rows / unit, chunks = (rows + most - 1) / most;
    return (units + chunks - 1) / chunks * unit;
}

// Seconds of one application on a CTA with `rows` rows: its FP64 instructions
// (a product and a sum each, 2.2 cycles of a partition per warp), a floor of
// one k's latency, and the norms and the barrier.
double app_seconds(int n, int rows, bool cplx, int cpt, int unit, int most, bool wide) {
    const int chunk = chunk_rows(rows, unit, most), chunks = (rows + chunk - 1) / chunk;
    const double steps = (double)(chunk / unit) * cpt;
    const double cycles = cplx ? std::max(42.0, 18.0 + 18.3 * steps) : std::max(42.0, 24.0 + 6.0 * steps);
    return chunks * (n * cycles / 1.9e9 + 0.4e-6 * steps / cpt) + (wide ? 3.6e-6 : 1.2e-6);
}

// The widest row ranges with which every matrix ends within `limit` alone.
void split_rows(const std::vector<int>& n, const std::vector<double>& apps, bool cplx, int cpt, int lanes, int unit,
                int most, double limit, Sched& sc, std::vector<double>& dur) {
    for (size_t k = 0; k < n.size(); ++k) {
        const int units = (n[k] + unit - 1) / unit;
        int lo = std::max(1, (units + lanes - 1) / lanes), hi = units;  // lo always taken, whatever its time
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (apps[k] * app_seconds(n[k], mid * unit, cplx, cpt, unit, most, mid < units) <= limit) lo = mid;
            else hi = mid - 1;
        }
        const int w = (units + lo - 1) / lo;
        const int u = (units + w - 1) / w;  // the same width, evenly
        sc.rows_per[k] = u * unit;
        sc.width[k] = (units + u - 1) / u;
        dur[k] = apps[k] * app_seconds(n[k], u * unit, cplx, cpt, unit, most, sc.width[k] > 1);
    }
}

// Longest first, onto the lanes that free up earliest.
void place(Sched& sc, const std::vector<double>& dur, int lanes) {
    const size_t cnt = dur.size();
    std::vector<int> order(cnt);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dur[x] > dur[y]; });
    std::vector<double> free_at(lanes, 0.0);
    struct Entry {
        double start;
        int seq, matrix, rank;
    };
    std::vector<std::vector<Entry>> per_lane(lanes);
    std::vector<int> idx(lanes);
    int seq = 0;
    sc.makespan = 0.0;
    for (int k : order) {
        const int w = sc.width[k];
        std::iota(idx.begin(), idx.end(), 0);
        std::partial_sort(idx.begin(), idx.begin() + w, idx.end(),
                          [&](int x, int y) { return free_at[x] < free_at[y] || (free_at[x] == free_at[y] && x < y); });
        double start = 0.0;
        for (int r = 0; r < w; ++r) start = std::max(start, free_at[idx[r]]);
        for (int r = 0; r < w; ++r) {
            per_lane[idx[r]].push_back(Entry{start, seq, k, r});
            free_at[idx[r]] = start + dur[k];
        }
        sc.makespan = std::max(sc.makespan, start + dur[k]);
        ++seq;
    }
    sc.offsets.assign(lanes + 1, 0);
    sc.plan.clear();
    for (int l = 0; l < lanes; ++l) {
        auto& v = per_lane[l];
        std::sort(v.begin(), v.end(), [](const Entry& x, const Entry& y) { return x.start < y.start || (x.start == y.start && x.seq < y.seq); });
        sc.offsets[l + 1] = sc.offsets[l] + (int)v.size();
        for (auto& e : v) sc.plan.push_back(TaylorPlan{e.matrix, e.rank});
    }
}

// Widths from a limit on each matrix's own time: the smallest limit with
// which all of them run side by side, found by bisection, and shorter ones,
// with which the later matrices follow on lanes that earlier ones left; the
// limit whose list schedule ends first is taken.
Sched schedule(const std::vector<int>& n, const std::vector<double>& apps, bool cplx, int cpt, int lanes, int unit, int most) {
    const size_t cnt = n.size();
    Sched sc, best;
    sc.width.assign(cnt, 1);
    sc.rows_per.assign(cnt, unit);
    std::vector<double> dur(cnt);
    double longest = 0.0;  // with one CTA each
    for (size_t k = 0; k < cnt; ++k)
        longest = std::max(longest, apps[k] * app_seconds(n[k], (n[k] + unit - 1) / unit * unit, cplx, cpt, unit, most, false));
    double lo = 0.0, hi = longest;
    for (int it = 0; it < 24; ++it) {
        const double mid = 0.5 * (lo + hi);
        split_rows(n, apps, cplx, cpt, lanes, unit, most, mid, sc, dur);
        if (std::accumulate(sc.width.begin(), sc.width.end(), 0) <= lanes) hi = mid;
        else lo = mid;
    }
    for (double f : {1.0, 0.8, 0.6, 0.4, 0.2}) {
        split_rows(n, apps, cplx, cpt, lanes, unit, most, hi * f, sc, dur);
        place(sc, dur, lanes);
        if (f == 1.0 || sc.makespan < best.makespan) best = sc;
        if (cnt == 1) break;
    }
    return best;
}

}  // namespace

void expmv_batch(Context& ctx, const std::vector<const DMat*>& as, const std::vector<const DMat*>& bs, double t,
                 std::vector<DMat>& results, std::vector<ExpmvInfo>& infos, int select_only_cols) {
    const size_t cnt = as.size();
    results.clear();
    results.resize(cnt);
    infos.assign(cnt, ExpmvInfo{});
    if (cnt == 0) return;
    const bool cplx = as[0]->cplx;
    const bool select_only = select_only_cols > 0;
    const int ncols = select_only ? select_only_cols : bs[0]->cols;
    for (size_t k = 0; k < cnt; ++k)
        if (as[k]->cplx != cplx || as[k]->rows < 1 ||
            (!select_only && (bs[k]->cols != ncols || bs[k]->rows != as[k]->rows)))
            fail(TNS_E_ARGUMENT, "internal: an exponential-action batch mixes element types or panel widths");

    // mu = trace / n (per part for complex), A - mu I, ||A - mu I||_1
    // (Expmv, :131-141; complex MatrixExponentialAction.Complex.cs:57-61; Dense, :157).
    std::vector<double> tr = traces(ctx, as);
    std::vector<DMat> sh(cnt);
    std::vector<double> mu_re(cnt), mu_im(cnt, 0.0);
    std::vector<const DMat*> shp(cnt);
    for (size_t k = 0; k < cnt; ++k) {
        const int n = as[k]->rows;
        mu_re[k] = tr[2 * k] / n;
        if (cplx) mu_im[k] = tr[2 * k + 1] / n;
        sh[k] = DMat(ctx, n, n, cplx, "the shifted operator");
        copy_dmat(ctx, sh[k], *as[k]);
        shift_diagonal(ctx, sh[k], -mu_re[k], cplx ? -mu_im[k] : 0.0);
        shp[k] = &sh[k];
    }
    std::vector<double> one_norm = norm1_batch(ctx, shp);

    // The sharp bounds d(p) = normest1(A^p)^(1/p), p = 2..9, for every matrix
    // outside condition 3.13 (:404-410): the search asks for all of them.
    const double scale = std::fabs(t);
    const double ca = 2.0 * kEll * kMaxPower * (kMaxPower + 3);
    const double cb = 9.9 / (ncols * 55.0);
    std::vector<size_t> sharp;
    std::vector<const DMat*> sharp_mats;
    for (size_t k = 0; k < cnt; ++k) {
        const double sn = scale * one_norm[k];
        if (sn != 0.0 && !(sn <= ca * cb)) {
            sharp.push_back(k);
            sharp_mats.push_back(shp[k]);
        }
    }
    std::vector<std::vector<double>> dp(cnt, std::vector<double>(kMaxPower + 2, std::numeric_limits<double>::quiet_NaN()));
    if (!sharp.empty()) {
        // Every (matrix, power) estimator of the batch advances together.
        std::vector<const DMat*> items;
        std::vector<int> powers;
        for (int p = 2; p <= kMaxPower + 1; ++p)
            for (const DMat* m : sharp_mats) {
                items.push_back(m);
                powers.push_back(p);
            }
        std::vector<double> v = power_norm_estimates(ctx, items, powers);
        size_t q = 0;
        for (int p = 2; p <= kMaxPower + 1; ++p)
            for (size_t k = 0; k < sharp.size(); ++k) dp[sharp[k]][p] = std::pow(v[q++], 1.0 / p);
    }

    // (m, s), eta and the coefficients, per matrix (Run, :258-283).
    std::vector<int> ms(cnt), ss(cnt);
    std::vector<double> eta_re(cnt), eta_im(cnt, 0.0);
    std::vector<double> coeffs;
    std::vector<size_t> coeff_off(cnt);
    for (size_t k = 0; k < cnt; ++k) {
        const double sn = scale * one_norm[k];
        int m = 0, s = 1;
        if (sn != 0.0) {
            const std::function<double(int)> alpha = [&](int p) { return net::max(dp[k][p], dp[k][p + 1]); };
            expmv_select_parameters(sn, &alpha, scale, ncols, m, s);
        }
        ms[k] = m;
        ss[k] = s;
        infos[k].degree = m;
        infos[k].scaling = s;
        if (!cplx) {
            eta_re[k] = std::exp((mu_re[k] * t) / (double)s);
        } else {
            net::Cx e = net::exp(net::div(net::Cx{mu_re[k] * t, mu_im[k] * t}, net::Cx{(double)s, 0.0}));
            eta_re[k] = e.re;
            eta_im[k] = e.im;
        }
        coeff_off[k] = coeffs.size();
        for (int j = 0; j < m; ++j) coeffs.push_back(t / (s * (double)(j + 1)));
    }

    if (select_only) return;
    if (ncols > 32) {
        // Wider panels than the fused kernel holds: the host-driven loop.
        for (size_t k = 0; k < cnt; ++k)
            expmv_taylor_host(ctx, sh[k], *bs[k], t, ms[k], ss[k], eta_re[k], eta_im[k], results[k], &infos[k]);
        return;
    }
    // The explicit zero skip only when some operator has a non-finite entry
    // (its parameters can still be finite: a nilpotent shifted operator has
    // d(p) = 0 for p >= 2).
    bool skip = false;
    for (size_t k = 0; k < cnt; ++k)
        if (!std::isfinite(one_norm[k])) skip = true;
    const Layout lay = taylor(ctx, cplx, skip, ncols, nullptr, 0);

    std::vector<int> orders(cnt);
    std::vector<double> apps(cnt);
    for (size_t k = 0; k < cnt; ++k) {
        orders[k] = as[k]->rows;
        apps[k] = std::max(1.0, (double)ms[k] * ss[k]);
    }
    Sched sc = schedule(orders, apps, cplx, ncols > 16 ? 2 : 1, lay.lanes, lay.unit, lay.rows);

    size_t panel_bytes = 0, slot_words = 0;
    for (size_t k = 0; k < cnt; ++k) {
        results[k] = DMat(ctx, orders[k], ncols, cplx, "the exponential action");
        panel_bytes += 2 * (size_t)orders[k] * lay.cols * as[k]->esz();
        slot_words += 6 * (size_t)sc.width[k];
    }
    DBuf panels(ctx, panel_bytes);
    const size_t state_bytes = sizeof(unsigned long long) + sizeof(int) * 2 * cnt;
    DBuf state(ctx, state_bytes);
    TNS_CUDA(cudaMemsetAsync(state.p, 0, state_bytes, ctx.stream));
    int* outs = reinterpret_cast<int*>(state.as<unsigned long long>() + 1);
    DBuf slots(ctx, sizeof(unsigned long long) * slot_words);
    TNS_CUDA(cudaMemsetAsync(slots.p, 0xff, sizeof(unsigned long long) * slot_words, ctx.stream));
    DBuf dcoeff(ctx, sizeof(double) * std::max<size_t>(coeffs.size(), 1));
    if (!coeffs.empty())
        TNS_CUDA(cudaMemcpyAsync(dcoeff.p, coeffs.data(), sizeof(double) * coeffs.size(), cudaMemcpyHostToDevice, ctx.stream));
    std::vector<TaylorDesc> descs(cnt);
    std::vector<CUtensorMap> maps(cnt);
    double* panel = panels.as<double>();
    unsigned long long* slot = slots.as<unsigned long long>();
    for (size_t k = 0; k < cnt; ++k) {
        TaylorDesc& d = descs[k];
        d.b = bs[k]->p;
        d.ldb = bs[k]->ld();
        d.f = results[k].p;
        const size_t es = cplx ? 2 : 1, panel_doubles = (size_t)orders[k] * lay.cols * es;
        d.w0 = panel;
        d.w1 = panel + panel_doubles;
        panel += 2 * panel_doubles;
        d.ldp = results[k].ld();
        d.coeff = dcoeff.as<double>() + coeff_off[k];
        d.slots = slot;
        slot += 6 * (size_t)sc.width[k];
        d.chunk = chunk_rows(sc.rows_per[k], lay.unit, lay.rows);
        encode_map_2d(&maps[k], sh[k].p, es * orders[k], orders[k], (uint64_t)sh[k].ld() * sh[k].esz(),
                      (uint32_t)(es * d.chunk), tile_k(d.chunk, lay.cols));
        d.out = outs + 2 * k;
        d.n = orders[k];
        d.m = ms[k];
        d.s = ss[k];
        d.width = sc.width[k];
        d.rows_per = sc.rows_per[k];
        d.eta_re = eta_re[k];
        d.eta_im = eta_im[k];
        d.eta_one = (eta_re[k] == 1.0 && eta_im[k] == 0.0) ? 1 : 0;
    }
    TaylorLaunch L{};
    UploadHold hold(ctx);  // the descriptors, the plan and its offsets
    L.descs = static_cast<const TaylorDesc*>(ctx.upload(descs.data(), sizeof(TaylorDesc) * cnt));
    L.plan = static_cast<const TaylorPlan*>(ctx.upload(sc.plan.data(), sizeof(TaylorPlan) * std::max<size_t>(sc.plan.size(), 1)));
    L.plan_off = static_cast<const int*>(ctx.upload(sc.offsets.data(), sizeof(int) * sc.offsets.size()));
    L.ncols = ncols;
    L.err = ctx.d_err;
    L.progress = state.as<unsigned long long>();
    // (A buffer of their own: beside the descriptors they could outgrow the upload ring.)
    DBuf dmaps(ctx, sizeof(CUtensorMap) * cnt);
    TNS_CUDA(cudaMemcpyAsync(dmaps.p, maps.data(), sizeof(CUtensorMap) * cnt, cudaMemcpyHostToDevice, ctx.stream));
    L.maps = dmaps.as<CUtensorMap>();
    taylor(ctx, cplx, skip, ncols, &L, lay.lanes);
    std::vector<int> h(2 * cnt);
    TNS_CUDA(cudaMemcpyAsync(h.data(), outs, sizeof(int) * 2 * cnt, cudaMemcpyDeviceToHost, ctx.stream));
    ctx.sync();
    for (size_t k = 0; k < cnt; ++k) {
        infos[k].applications = h[2 * k];
        infos[k].early_exits = h[2 * k + 1];
    }
}

void expmv(Context& ctx, const DMat& a, const DMat& b, double t, DMat& result, ExpmvInfo* info) {
    std::vector<const DMat*> as{&a}, bs{&b};
    std::vector<DMat> res;
    std::vector<ExpmvInfo> infs;
    expmv_batch(ctx, as, bs, t, res, infs);
    result = std::move(res[0]);
    if (info) *info = infs[0];
}

}  // namespace tns
