// LU panel factorization with the panel's rows in registers, spread over a
// thread-block cluster.
//
// getf2 on an m x 32 panel (Lu.cs:384-424, BlockedLu.cs:148-200): per column
// the pivot is the first row of the largest measure (|a|, or |Re| + |Im|),
// rows j and p change places, the column is scaled by the pivot's reciprocal
// (divided when |pivot| < SafeMin) and the later columns take the rank-1
// update t + (-u) l with two roundings. It is a chain of 32 dependent column
// steps, so its time is the latency of one step, not the m w^2 operations.
//
// Layout. One thread holds one row in registers for the whole panel; a panel
// taller than one CTA's threads is spread over the CTAs of a cluster (up to
// eight). The rows never move: a thread keeps the position its row currently
// has, an interchange changes two positions, and every row is written to its
// final position once at the end. The registers shift by one column per step
// (column j is always a[0]), so the step is a loop with static register
// indices; the working width drops by 8 every 8 steps (608 column updates
// per row instead of the triangle's 496, in code small enough for the
// instruction cache -- a fully unrolled 32-column step is not).
//
// One step. Each warp finds its best row with one integer warp reduction of the
// measure's leading word (the bit patterns are ordered as the values; NaNs
// count as no candidate, as in the reference's comparison; the trailing word
// and the position are only compared on ties) and puts its measure and position
// in shared memory; after a block barrier every warp folds the block's
// candidates to the same winner, whose lane writes its row. A panel in one
// CTA then has its pivot row. In a group, the winner's warp sends key and row
// to every CTA
// of the group by st.async through distributed shared memory, counted in
// bytes on the receiver's mbarrier, so the exchange needs no cluster-wide
// fence (an mbarrier arrival with release.cluster semantics measured 700
// cycles here). All buffers alternate by column parity: a warp reuses one only
// after a block barrier, a sender only after the receiver's answer, for the
// column in between.
//
// Batches. The host packs the panels of a batch into clusters (a group of
// ceil(rows / threads) CTAs per panel, several groups per cluster when they
// fit), so one launch serves panels of any heights. Every wait is bounded; all
// CTAs of a cluster meet once at the end, so none leaves while another may
// still read its shared memory.

#include "lu_panel.h"

#include <algorithm>
#include <atomic>
#include <climits>
#include <numeric>

#include "batch.cuh"
#include "device_util.cuh"
#include "tcgen05.cuh"

namespace tns {

namespace {

constexpr double kSafeMin = 2.2250738585072014e-308;
constexpr int kW = kRowPanelWidth;
constexpr int kRow = kW + 2;          // a candidate row in shared memory: its entries, its position, padding
constexpr int kMaxCluster = 8;       // portable cluster size
constexpr int kNoRow = INT_MAX;      // position of a thread without a row
constexpr int kErrRowPanel = 22;     // a group's exchange was waited for in vain

// Largest CTA: a row of 32 columns is 64 registers real, 128 complex, beside
// about 50 others, out of 65,536 / threads.
template <bool CPLX>
constexpr int kMaxThreads = CPLX ? 256 : 512;

struct PanelSlot {
    int item;        // -1: no work for this CTA
    int rank, size;  // this CTA's place in its panel's group
    int base;        // cluster rank of the group's first CTA
};

template <bool CPLX>
struct El;
template <>
struct El<false> {
    using T = double;
    static __device__ __forceinline__ double measure(double v) {
        return __longlong_as_double(__double_as_longlong(v) & 0x7fffffffffffffffll);
    }
    static __device__ __forceinline__ bool nonzero(double v) { return v != 0.0; }
    // t + (-u) l, two roundings
    static __device__ __forceinline__ double update(double t, double u, double l) { return add_rn(t, mul_rn(-u, l)); }
};
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(sub_rn(mul_rn(a.x, b.x), mul_rn(a.y, b.y)), add_rn(mul_rn(a.y, b.x), mul_rn(a.x, b.y)));
}
// Smith's division, as System.Numerics.Complex divides.
__device__ __forceinline__ double2 cdiv(double2 l, double2 r) {
    const double a = l.x, b = l.y, c = r.x, d = r.y;
    if (fabs(d) < fabs(c)) {
        const double doc = __ddiv_rn(d, c);
        const double den = add_rn(c, mul_rn(d, doc));
        return make_double2(__ddiv_rn(add_rn(a, mul_rn(b, doc)), den), __ddiv_rn(sub_rn(b, mul_rn(a, doc)), den));
    }
    const double cod = __ddiv_rn(c, d);
    const double den = add_rn(d, mul_rn(c, cod));
    return make_double2(__ddiv_rn(add_rn(b, mul_rn(a, cod)), den), __ddiv_rn(add_rn(-a, mul_rn(b, cod)), den));
}
template <>
struct El<true> {
    using T = double2;
    static __device__ __forceinline__ double measure(double2 v) { return add_rn(fabs(v.x), fabs(v.y)); }
    static __device__ __forceinline__ bool nonzero(double2 v) { return !(v.x == 0.0 && v.y == 0.0); }
    static __device__ __forceinline__ double2 update(double2 t, double2 u, double2 l) {
        const double2 p = cmul(make_double2(-u.x, -u.y), l);
        return make_double2(add_rn(t.x, p.x), add_rn(t.y, p.y));
    }
};

// The scaling of a column by its pivot: a product with the reciprocal, or a
// division when |pivot| < SafeMin (Lu.cs:409-412, BlockedLu.cs:175-183).
template <bool CPLX>
struct Scale;
template <>
struct Scale<false> {
    double value, r;
    bool zero, recip;
    __device__ __forceinline__ explicit Scale(double v) {
        value = v;
        r = __ddiv_rn(1.0, v);
        zero = v == 0.0;
        recip = fabs(v) >= kSafeMin;
    }
    __device__ __forceinline__ double operator()(double l) const {
        if (zero) return l;
        return recip ? mul_rn(l, r) : __ddiv_rn(l, value);
    }
};
template <>
struct Scale<true> {
    double2 value, r;
    bool zero, recip;
    // Every lane of the warp passes the same v. 1 / v by Smith's division (cdiv
    // of (1, 0)), its two branches on one path and its two quotients, which
    // share the divisor, one each in the even and the odd lanes: two division
    // latencies instead of three (the column step waits for this value).
    __device__ __forceinline__ explicit Scale(double2 v) {
        value = v;
        zero = v.x == 0.0 && v.y == 0.0;
        // The modulus is at least the larger part, so a part of SafeMin or
        // more decides without forming it.
        recip = fabs(v.x) >= kSafeMin || fabs(v.y) >= kSafeMin || cabs_net(v.x, v.y) >= kSafeMin;
        const bool re_larger = fabs(v.y) < fabs(v.x);
        const double big = re_larger ? v.x : v.y, small = re_larger ? v.y : v.x;
        const double ratio = __ddiv_rn(small, big);
        const double den = add_rn(big, mul_rn(small, ratio));
        const double zr = mul_rn(0.0, ratio), or_ = mul_rn(1.0, ratio);
        const double num_re = re_larger ? add_rn(1.0, zr) : add_rn(0.0, or_);
        const double num_im = re_larger ? sub_rn(0.0, or_) : add_rn(-1.0, zr);
        const bool odd = threadIdx.x & 1;
        const double mine = __ddiv_rn(odd ? num_im : num_re, den);
        const double other = __shfl_xor_sync(0xffffffffu, mine, 1);
        r = odd ? make_double2(other, mine) : make_double2(mine, other);
    }
    __device__ __forceinline__ double2 operator()(double2 l) const {
        if (zero) return l;
        return recip ? cmul(l, r) : cdiv(l, value);
    }
};

// Stores to shared memory of a cluster CTA that complete `bar` there by their
// bytes. Addresses are shared::cluster ones.
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, double2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, ulonglong2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "l"(v.x), "l"(v.y), "r"(bar)
                 : "memory");
}
// Bounded wait for a phase completed by other CTAs of the cluster (acquire at
// cluster scope).
__device__ __forceinline__ bool wait_cluster(uint64_t* bar, uint32_t parity, int* err) {
    auto ready = [&] {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        return ok != 0;
    };
    if (ready()) return true;
    const unsigned long long start = global_timer_ns();
    for (uint32_t it = 1;; ++it) {
        if (ready()) return true;
        if ((it & 255u) == 0) {
            if (*reinterpret_cast<volatile int*>(err) != 0) return false;
            if (global_timer_ns() - start > kWaitTimeoutNs) {
                atomicCAS(err, 0, kErrRowPanel);
                return false;
            }
        }
    }
}

// The order of the pivot search as an unsigned key: larger measures larger,
// 0 for a NaN (never a candidate) -- the measure's bits plus one, its sign bit
// being clear. Integer arithmetic throughout: its latency is half of the FP64
// pipe's.
__device__ __forceinline__ unsigned long long measure_key(double m, bool active) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(m);
    return active && bits <= 0x7ff0000000000000ull ? bits + 1 : 0ull;
}

// The lanes holding the best of a warp's (key, position) pairs, as a mask of
// one bit (of several only when no lane has a row): the largest key, the lowest
// position on ties. The same in every lane.
__device__ __forceinline__ unsigned warp_pick(unsigned long long key, int pos) {
    const unsigned full = 0xffffffffu;
    const uint32_t hi = (uint32_t)(key >> 32), lo = (uint32_t)key;
    bool eq = hi == __reduce_max_sync(full, hi);
    unsigned who = __ballot_sync(full, eq);
    if (who & (who - 1)) {  // a tie in the leading word
        const uint32_t best_lo = __reduce_max_sync(full, eq ? lo : 0u);  // every lane takes part
        eq = eq && lo == best_lo;
        const uint32_t best_pos = __reduce_min_sync(full, (uint32_t)(eq ? pos : kNoRow));
        eq = eq && (uint32_t)pos == best_pos;
        who = __ballot_sync(full, eq);
    }
    return who;
}

// The first NC entries of a row to shared memory (16-byte aligned), in 16-byte
// stores.
template <int NC>
__device__ __forceinline__ void store_row(double* dst, const double (&a)[kW]) {
#pragma unroll
    for (int c = 0; c < NC; c += 2) *reinterpret_cast<double2*>(dst + c) = make_double2(a[c], a[c + 1]);
}
template <int NC>
__device__ __forceinline__ void store_row(double2* dst, const double2 (&a)[kW]) {
#pragma unroll
    for (int c = 0; c < NC; ++c) dst[c] = a[c];
}

template <bool CPLX>
struct PanelState {
    using E = typename El<CPLX>::T;
    E* save;  // this thread's finished entries: save[c * T]
    // Candidate rows and their positions by parity: [2][kRow] this CTA's, then
    // [2][kMaxCluster][kRow] the group's.
    E* cand;
    ulonglong2* keys;   // [2][32] this CTA's candidates: measure key, position
    ulonglong2* gkeys;  // [2][kMaxCluster] the group's
    uint64_t* bars;     // [2]
    int T, warps, rank, size, base, w, limit, r0;
    int* piv;
    int* singular;
    int* err;
};

// Up to eight column steps with a working width of NC columns, from column
// j0. False: a wait gave up.
template <bool CPLX, int NC>
__device__ __forceinline__ bool panel_phase(const PanelState<CPLX>& s, typename El<CPLX>::T (&a)[kW], int& pos, int j0) {
    using E = typename El<CPLX>::T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jend = min(j0 + 8, s.limit);
#pragma unroll 1
    for (int j = j0; j < jend; ++j) {
        const int par = j & 1;
        // This warp's candidate.
        const bool active = pos != kNoRow && pos >= j;
        const unsigned long long key = measure_key(El<CPLX>::measure(a[0]), active);
        const unsigned mine = warp_pick(key, active ? pos : kNoRow);
        const bool candidate = (mine & (0u - mine)) == 1u << lane;
        if (candidate)
            s.keys[par * 32 + warp] = make_ulonglong2(key, (unsigned long long)(unsigned)(active ? pos : kNoRow));
        __syncthreads();
        // The block's winner, the same in every warp; its warp publishes the row
        // and, behind it, the row's position.
        ulonglong2 k = make_ulonglong2(0ull, (unsigned long long)(unsigned)kNoRow);
        if (lane < s.warps) k = s.keys[par * 32 + lane];
        unsigned won = warp_pick(k.x, (int)k.y);
        const bool block_won = (won & (0u - won)) == 1u << warp;
        int at = par * kRow;  // the pivot row's place in cand
        bool here = true;     // the pivot row is this CTA's
        if (block_won && candidate) {
            store_row<NC>(s.cand + at, a);
            *reinterpret_cast<int*>(s.cand + at + kW) = active ? pos : kNoRow;
        }
        if (s.size == 1) {
            __syncthreads();
        } else {
            const int rows_at = (2 + par * kMaxCluster) * kRow;
            if (threadIdx.x == 0)
                mbar_arrive_expect_tx(&s.bars[par], (uint32_t)(s.size * ((NC + 1) * (int)sizeof(E) + 16)));
            if (block_won) {
                __syncwarp();
                const int e = lane < NC ? lane : kW;  // a row entry per lane, the position in lane NC (or, of 32, after)
                const E v = s.cand[at + e];
                const ulonglong2 kw = make_ulonglong2(__shfl_sync(0xffffffffu, k.x, warp), __shfl_sync(0xffffffffu, k.y, warp));
                for (int r = 0; r < s.size; ++r) {
                    const uint32_t cta = (uint32_t)(s.base + r), bar = cluster_addr(&s.bars[par], cta);
                    if (lane < NC || (NC < 32 && lane == NC))
                        st_async(cluster_addr(s.cand + rows_at + s.rank * kRow + e, cta), v, bar);
                    if (lane == 0) {
                        if (NC == 32) st_async(cluster_addr(s.cand + rows_at + s.rank * kRow + kW, cta), s.cand[at + kW], bar);
                        st_async(cluster_addr(s.gkeys + par * kMaxCluster + s.rank, cta), kw, bar);
                    }
                }
            }
            const bool got = wait_cluster(&s.bars[par], (uint32_t)((j >> 1) & 1), s.err);
            if (!__syncthreads_and(got)) return false;
            k = make_ulonglong2(0ull, (unsigned long long)(unsigned)kNoRow);
            if (lane < s.size) k = s.gkeys[par * kMaxCluster + lane];
            won = warp_pick(k.x, (int)k.y);
            const int owner = __ffs(won) - 1;
            at = rows_at + owner * kRow;
            here = owner == s.rank;
        }
        const E* u = s.cand + at;
        const int p = *reinterpret_cast<const int*>(u + kW);
        // Columns with a zero in the pivot row are skipped, as the reference
        // skips them; the checks only run where the row has one.
        const bool some_zero = lane > 0 && lane < NC && j + lane < s.w && !El<CPLX>::nonzero(u[lane]);
        const bool checked = __any_sync(0xffffffffu, some_zero);
        const Scale<CPLX> scale(u[0]);
        if (s.rank == 0 && threadIdx.x == 0) {
            s.piv[s.r0 + j] = s.r0 + p;
            if (scale.zero) atomicMin(s.singular, s.r0 + j);
        }
        // The pivot row is finished: its warp keeps it, a lane per column.
        if (here && block_won && lane < NC && j + lane < s.w)
            s.save[(size_t)(j + lane) * s.T + (__ffs(mine) - 1 - lane)] = u[lane];
        // The interchange: two rows change positions.
        if (pos == p) pos = j;
        else if (pos == j) pos = p;
        if (pos != kNoRow && pos > j) {
            const E l = scale(a[0]);
            s.save[(size_t)j * s.T] = l;
            if (!checked) {
#pragma unroll
                for (int c = 1; c < NC; ++c) a[c - 1] = El<CPLX>::update(a[c], u[c], l);
            } else {
#pragma unroll
                for (int c = 1; c < NC; ++c) {
                    const E uc = u[c];
                    a[c - 1] = El<CPLX>::nonzero(uc) ? El<CPLX>::update(a[c], uc, l) : a[c];
                }
            }
        }
    }
    return true;
}

template <bool CPLX>
__global__ void __launch_bounds__(kMaxThreads<CPLX>, 1)
    row_panel_kernel(const __grid_constant__ Batch<PanelFactorDesc> b, const PanelSlot* __restrict__ slots, int* err) {
    using E = typename El<CPLX>::T;
    extern __shared__ __align__(16) unsigned char panel_smem[];
    __shared__ __align__(16) ulonglong2 s_keys[2 * 32];
    __shared__ __align__(16) ulonglong2 s_gkeys[2 * kMaxCluster];
    __shared__ __align__(8) uint64_t s_bars[2];
    const int T = blockDim.x, warps = T >> 5, tid = threadIdx.x;
    PanelSlot sl;
    if (slots) {
        sl = slots[blockIdx.x];
    } else {
        sl.item = 0;
        sl.rank = (int)cluster_ctarank();
        sl.size = (int)gridDim.x;  // one panel: one cluster
        sl.base = 0;
    }
    if (tid == 0) {
        mbar_init(&s_bars[0], 1);
        mbar_init(&s_bars[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    cluster_sync();  // every CTA's barriers exist before another reaches them
    // A carried row that moves: its entries, read before any is written.
    E moved[kW];
    E* carried = nullptr;
    int ld = 0, carry = 0;
    if (sl.item >= 0) {
        const PanelFactorDesc& d = batch_item(b, sl.item);
        PanelState<CPLX> s;
        E* sm = reinterpret_cast<E*>(panel_smem);
        s.save = sm + tid;             // [kW][T]
        s.cand = sm + (size_t)kW * T;  // [2][kRow], [2][kMaxCluster][kRow]
        s.keys = s_keys;
        s.gkeys = s_gkeys;
        s.bars = s_bars;
        s.T = T;
        s.warps = warps;
        s.rank = sl.rank;
        s.size = sl.size;
        s.base = sl.base;
        const int M = d.m - d.r0;
        s.w = d.w;
        s.limit = min(M, d.w);
        s.r0 = d.r0;
        s.piv = d.piv;
        s.singular = d.singular;
        s.err = err;
        E* P = reinterpret_cast<E*>(d.a) + (size_t)d.r0 * d.ld + d.r0;  // panel origin
        const int row = sl.rank * T + tid;
        int pos = row < M ? row : kNoRow;
        E a[kW];
#pragma unroll
        for (int c = 0; c < kW; ++c) {
            a[c] = E{};
            if (row < M && c < d.w) a[c] = P[(size_t)c * d.ld + row];
        }
        bool ok = panel_phase<CPLX, 32>(s, a, pos, 0);
        if (ok && s.limit > 8) ok = panel_phase<CPLX, 24>(s, a, pos, 8);
        if (ok && s.limit > 16) ok = panel_phase<CPLX, 16>(s, a, pos, 16);
        if (ok && s.limit > 24) ok = panel_phase<CPLX, 8>(s, a, pos, 24);
        // A pivot row's entries were stored by the lanes of its warp; after the
        // last column no block barrier lies between that and reading them here.
        __syncwarp();
        if (ok && row < M) {
            for (int c = 0; c < d.w; ++c) P[(size_t)c * d.ld + pos] = s.save[(size_t)c * T];
            if (d.carry > 0 && pos != row) {
                ld = d.ld;
                carry = d.carry;
                const E* from = P - (size_t)carry * ld + row;
                carried = P - (size_t)carry * ld + pos;
#pragma unroll
                for (int c = 0; c < kW; ++c)
                    if (c < carry) moved[c] = from[(size_t)c * ld];
            }
        }
    }
    // Nobody leaves while a peer's stores may still be on their way to it, and
    // no carried entry is written before all are read.
    cluster_sync();
    if (carried) {
#pragma unroll
        for (int c = 0; c < kW; ++c)
            if (c < carry) carried[(size_t)c * ld] = moved[c];
    }
}

// Shared memory of one CTA: the finished entries and both parities' candidate
// rows, the block's and the group's.
size_t row_panel_smem(bool cplx, int threads) {
    const size_t es = cplx ? 16 : 8;
    return es * (kW * (size_t)threads + 2 * (1 + kMaxCluster) * kRow);
}

template <bool CPLX>
void launch(Context& ctx, const std::vector<PanelFactorDesc>& v) {
    // The fewest CTAs per panel, evenly filled. More and smaller ones shorten
    // the updates but cost the exchange (about 700 cycles a column): at 512 rows
    // one real CTA of 512 threads measured 37 us against 43 us for four of 128,
    // and two complex ones of 256 60 us against 54 us for four of 128, while a
    // batch wants its SMs for other panels.
    const int top = kMaxThreads<CPLX>;
    int rows_max = 0;
    for (auto& p : v) rows_max = std::max(rows_max, p.m - p.r0);
    const int cs = std::max(1, (rows_max + top - 1) / top);
    const int threads = round_up((rows_max + cs - 1) / cs, 32);
    if (cs > kMaxCluster) fail(TNS_E_ARGUMENT, "internal: panel too tall for the register kernel");
    UploadHold hold(ctx);  // the slots and the panels
    const PanelSlot* d_slots = nullptr;
    int grid = cs;
    if (v.size() > 1) {
        // Groups into clusters of cs CTAs, tallest first.
        std::vector<int> order(v.size());
        std::iota(order.begin(), order.end(), 0);
        auto size_of = [&](int i) { return std::max(1, (v[i].m - v[i].r0 + threads - 1) / threads); };
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return size_of(x) > size_of(y); });
        // Each into the fullest cluster that has room for it.
        std::vector<PanelSlot> slots;
        std::vector<int> open[kMaxCluster];  // clusters by their free CTAs
        for (int i : order) {
            const int g = size_of(i);
            int left = g;
            while (left < cs && open[left].empty()) ++left;
            size_t k = slots.size() / cs;
            if (left < cs) {
                k = open[left].back();
                open[left].pop_back();
            } else {
                slots.resize(slots.size() + cs, PanelSlot{-1, 0, 0, 0});
            }
            for (int r = 0; r < g; ++r) slots[k * cs + cs - left + r] = PanelSlot{i, r, g, cs - left};
            if (left > g) open[left - g].push_back((int)k);
        }
        grid = (int)slots.size();
        d_slots = static_cast<const PanelSlot*>(ctx.upload(slots.data(), sizeof(PanelSlot) * slots.size()));
    }
    const size_t smem = row_panel_smem(CPLX, threads);
    static std::atomic<bool> configured[64];
    if (!configured[ctx.device].load(std::memory_order_acquire)) {
        TNS_CUDA(cudaFuncSetAttribute(row_panel_kernel<CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)row_panel_smem(CPLX, top)));
        configured[ctx.device].store(true, std::memory_order_release);
    }
    Batch<PanelFactorDesc> b = make_batch(ctx, v);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TNS_CUDA(cudaLaunchKernelEx(&cfg, row_panel_kernel<CPLX>, b, d_slots, ctx.d_err));
    ctx.kernel_launches++;
}

// ---- interchanges and U12 -------------------------------------------------------
//
// After a panel, every other column takes the panel's row interchanges and, to
// the right of it, U12 := L11^-1 A12 (Triangular.SolveLowerUnit,
// Triangular.cs:26-57; BlockedLu.cs:312-327). One warp per column does both in one
// pass: every CTA turns the interchanges into moves (which row each touched
// position ends up with, by following the swaps' references in parallel), the
// warp loads all of a column's moved rows at once and stores them at their
// places, and the top w, already in its lanes, go through the triangle first.
// One thread per column swapping rows in turn took 26 us a step at n = 512, its
// loads and stores one dependent chain through L2, and the triangle a launch of
// its own after it.

constexpr int kRowsWarps = 8;

struct PanelMoves {
    int p[kPanelRowsMaxWidth];      // the swaps' partners
    int root[kPanelRowsMaxWidth];   // the swap whose own row holds what swap s's own position holds before it
    int prev[kPanelRowsMaxWidth];   // the latest earlier swap with the same partner, or -1
    int top[kPanelRowsMaxWidth];    // the row that ends at position k0 + s
    int dst[kPanelRowsMaxWidth];    // a position beyond the panel's rows that swap s is the last to touch, or -1
    int src[kPanelRowsMaxWidth];    // and the row that ends there
};

// Swap s exchanges positions r_s = k0 + s and p_s >= r_s. What r_s holds just
// before is what the latest earlier swap with partner r_s brought there -- the
// values its own position held before it, and so on back to a position no swap
// had touched. Position r_s ends with what p_s holds before swap s; a partner
// beyond the panel's rows ends with what its last swap's own position held.
__device__ __forceinline__ void panel_moves(PanelMoves& M, const PanelRowsDesc& d) {
    const int s = threadIdx.x, w = d.w;
    if (s < w) M.p[s] = d.swap ? d.piv[d.k0 + s] : d.k0 + s;
    __syncthreads();
    int link = -1, prev = -1;
    bool last = true;
    const int r = d.k0 + s, p = s < w ? M.p[s] : 0;
    const bool real = s < w && p != r;
    if (s < w) {
        for (int q = 0; q < w; ++q) {
            const int pq = M.p[q];
            if (pq == d.k0 + q) continue;  // no swap
            if (q < s && pq == r) link = q;
            if (q < s && pq == p) prev = q;
            if (q > s && pq == p) last = false;
        }
        M.root[s] = link < 0 ? s : link;
        M.prev[s] = prev;
    }
    __syncthreads();
    // Pointer jumping: chains of at most w links.
    for (int reach = 1; reach < w; reach *= 2) {
        const int next = s < w ? M.root[M.root[s]] : 0;
        __syncthreads();
        if (s < w) M.root[s] = next;
        __syncthreads();
    }
    if (s < w) {
        const int own = d.k0 + M.root[s];
        M.top[s] = !real ? own : M.prev[s] >= 0 ? d.k0 + M.root[M.prev[s]] : p;
        M.dst[s] = real && last && p >= d.k0 + w ? p : -1;
        M.src[s] = own;
    }
    __syncthreads();
}

template <bool CPLX>
__global__ void __launch_bounds__(32 * kRowsWarps) panel_rows_kernel(const __grid_constant__ Batch<PanelRowsDesc> b,
                                                                    int cols_per_cta) {
    using El_ = El<CPLX>;
    using E = typename El_::T;
    int lo = 0, hi = b.count - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (batch_item(b, mid).tile_begin <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const PanelRowsDesc& d = batch_item(b, lo);
    extern __shared__ __align__(16) unsigned char panel_smem[];
    E* t = reinterpret_cast<E*>(panel_smem);  // t[k * w + i] = L11(i, k)
    __shared__ PanelMoves M;
    const int w = d.w, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    E* a = reinterpret_cast<E*>(d.a);
    if (d.solve)
        for (int e = threadIdx.x; e < w * w; e += 32 * kRowsWarps) {
            const int k = e / w, i = e - k * w;
            t[e] = a[(size_t)(d.k0 + k) * d.ld + d.k0 + i];
        }
    panel_moves(M, d);  // ends with a block barrier: the triangle is there too
    const int first = d.c0 + ((int)blockIdx.x - d.tile_begin) * cols_per_cta;
    for (int c = first + warp; c < min(d.c1, first + cols_per_cta); c += kRowsWarps) {
        E* col = a + (size_t)c * d.ld;
        E v[2], out[2];
        int dst[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int s = lane + 32 * h;
            dst[h] = -1;
            v[h] = E{};
            if (s < w) {
                v[h] = col[M.top[s]];
                dst[h] = M.dst[s];
                if (dst[h] >= 0) out[h] = col[M.src[s]];
            }
        }
        __syncwarp();  // every row is read before one is written
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (dst[h] >= 0) col[dst[h]] = out[h];
        if (d.solve) {
            auto pick = [](bool c1, E x, E y) { return c1 ? x : y; };
            auto bcast = [](E x, int src) {
                if constexpr (CPLX) return make_double2(__shfl_sync(0xffffffffu, x.x, src), __shfl_sync(0xffffffffu, x.y, src));
                else return __shfl_sync(0xffffffffu, x, src);
            };
#pragma unroll 4
            for (int k = 0; k < min(w, 32); ++k) {
                const E x = bcast(v[0], k);
                const bool nz = El_::nonzero(x);
                v[0] = pick(nz & (lane > k) & (lane < w), El_::update(v[0], x, t[k * w + min(lane, w - 1)]), v[0]);
                if (w > 32) v[1] = pick(nz & (lane + 32 < w), El_::update(v[1], x, t[k * w + min(lane + 32, w - 1)]), v[1]);
            }
#pragma unroll 4
            for (int k = 32; k < w; ++k) {
                const E x = bcast(v[1], k - 32);
                v[1] = pick(El_::nonzero(x) & (lane + 32 > k) & (lane + 32 < w),
                            El_::update(v[1], x, t[k * w + min(lane + 32, w - 1)]), v[1]);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (lane + 32 * h < w) col[d.k0 + lane + 32 * h] = v[h];
    }
}

template <bool CPLX>
void launch_rows(Context& ctx, std::vector<PanelRowsDesc>& v) {
    long long cols = 0;
    int wmax = 0;
    for (auto& d : v) {
        cols += d.c1 - d.c0;
        if (d.solve) wmax = std::max(wmax, d.w);
    }
    // A column per warp until the grid is four CTAs per SM; then more.
    const int per = kRowsWarps * (int)std::max(1LL, cols / (4LL * kRowsWarps * ctx.num_sms));
    long long total = 0;
    for (auto& d : v) {
        d.tile_begin = (int)total;
        total += (d.c1 - d.c0 + per - 1) / per;
    }
    const size_t es = CPLX ? 16 : 8, smem = es * wmax * wmax;
    static std::atomic<bool> configured[64];
    if (!configured[ctx.device].load(std::memory_order_acquire)) {
        TNS_CUDA(cudaFuncSetAttribute(panel_rows_kernel<CPLX>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(es * kPanelRowsMaxWidth * kPanelRowsMaxWidth)));
        configured[ctx.device].store(true, std::memory_order_release);
    }
    panel_rows_kernel<CPLX><<<(unsigned)total, 32 * kRowsWarps, smem, ctx.stream>>>(make_batch(ctx, v), per);
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
}

}  // namespace

int row_panel_max_rows(bool cplx) {
    return kMaxCluster * (cplx ? kMaxThreads<true> : kMaxThreads<false>);
}

void launch_row_panels(Context& ctx, bool cplx, const std::vector<PanelFactorDesc>& v) {
    if (v.empty()) return;
    if (cplx) launch<true>(ctx, v);
    else launch<false>(ctx, v);
}

void launch_panel_rows(Context& ctx, bool cplx, std::vector<PanelRowsDesc>& v) {
    std::vector<PanelRowsDesc> live;
    for (auto& d : v)
        if (d.c1 > d.c0 && d.w > 0 && (d.swap || d.solve)) live.push_back(d);
    if (live.empty()) return;
    if (cplx) launch_rows<true>(ctx, live);
    else launch_rows<false>(ctx, live);
}

}  // namespace tns
