// The kernels behind the norm estimates of a matrix's powers: the estimator's
// products A X and A^H X with one or two columns, and the ell test's chain
// ||abs(A)^p||_1. Both are sequences of n-term sums in a prescribed order, so a
// result's time is the length of its sum times the latency of an addition
// (8 cycles), as long as the loads run far enough ahead; these kernels are laid
// out for that.

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "batch.cuh"
#include "device_util.cuh"
#include "tcgen05.cuh"
#include "tns_internal.h"

namespace tns {

namespace {

// Asynchronous copies global -> shared; an invalid one fills with zeros.
__device__ __forceinline__ void cp16(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp8(void* dst, const void* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ bool is_zero(double v) { return (__double_as_longlong(v) << 1) == 0; }

// ---- Y := A X, X n x t, t <= 2 -----------------------------------------------
// The axpy order of PanelProduct.Apply (PanelProduct.cs:25-41): y[i] accumulates
// x[j] * a[i, j] for j = 0..n-1, two roundings per term, terms of a zero x[j]
// left out (a skipped term adds +0 to a sum that is never -0). Complex operator
// (LinearOperators.cs:262-282): pr = Ar xr, pi = Ar xi, qr = Ai xr, qi = Ai xi,
// then (pr - qi, pi + qr).
//
// One warp per CTA: its 32 lanes are 128 bytes of rows (8 complex, 16 real) by
// the row's independent sums -- complex: the two columns' real and imaginary x,
// each lane two sums -- so every SM gets a few of these short chains (n = 512
// complex: 64 CTAs; a thread per (row, column) and 64 rows per CTA used eight
// SMs). A and x arrive by cp.async in tiles of kApplyK columns, kApplyStages - 1
// of them in flight: 24 KB, what the chain consumes in the latency of HBM.
// Four FP64 instructions per step and lane (8.8 cycles of the pipe) cover the
// addition's latency.
constexpr int kApplyK = 16;
constexpr int kApplyStages = 12;

template <bool CPLX>
struct ApplyTile {
    static constexpr int ROWS = CPLX ? 8 : 16;
    double a[kApplyK][16];                // [k][row (re, im)]
    double x[2][kApplyK * (CPLX ? 2 : 1)];  // [column][k (re, im)]
};

template <bool CPLX>
__global__ void __launch_bounds__(32) power_apply_kernel(const __grid_constant__ Batch<PanelDesc> b) {
    using Tile = ApplyTile<CPLX>;
    constexpr int ES = CPLX ? 2 : 1;
    const PanelDesc& d = batch_item(b, blockIdx.y);
    const int n = d.n, t = d.t, i0 = blockIdx.x * Tile::ROWS;
    if (i0 >= n) return;
    extern __shared__ __align__(128) unsigned char apply_smem[];
    Tile* ring = reinterpret_cast<Tile*>(apply_smem);
    const int lane = threadIdx.x;
    const int tiles = (n + kApplyK - 1) / kApplyK;
    // The matrix is padded with zeros to multiples of 64 rows and columns, so a
    // tile's rows and columns past n may be read.
    auto stage = [&](int q) {
        if (q < tiles) {
            Tile& T = ring[q % kApplyStages];
            const int k0 = q * kApplyK;
#pragma unroll
            for (int e = lane; e < kApplyK * 8; e += 32) {
                const int k = e >> 3, c = e & 7;  // 16-byte piece c of column k0 + k
                cp16(&T.a[k][c * 2], d.a + ((size_t)(k0 + k) * d.ld + i0) * ES + c * 2, true);
            }
            if constexpr (CPLX) {
                const int c = lane >> 4, k = lane & 15;
                const bool ok = c < t && k0 + k < n;
                cp16(&T.x[c][2 * k], ok ? d.x + ((size_t)c * d.ldx + k0 + k) * 2 : d.x, ok);
            } else {
                const int c = lane >> 4, k = lane & 15;
                const bool ok = c < t && k0 + k < n;
                cp8(&T.x[c][k], ok ? d.x + (size_t)c * d.ldx + k0 + k : d.x, ok);
            }
        }
        cp_commit();
    };
    for (int q = 0; q < kApplyStages - 1; ++q) stage(q);
    // Complex: row = lane & 7, x part = bit 3, column = bit 4; real: row = lane &
    // 15, column = bit 4.
    const int row = lane & (Tile::ROWS - 1), part = CPLX ? (lane >> 3) & 1 : 0, col = lane >> 4;
    double p = 0.0, q_ = 0.0;
    for (int q = 0; q < tiles; ++q) {
        cp_wait<kApplyStages - 2>();
        __syncwarp();
        stage(q + kApplyStages - 1);  // into the slot finished last trip
        const Tile& T = ring[q % kApplyStages];
        const int len = min(kApplyK, n - q * kApplyK);
        // Zeros among the tile's x (all its columns and parts)?
        bool zero;
        if constexpr (CPLX) {
            const int k = lane & 15;
            zero = (lane >> 4) < t && k < len && (is_zero(T.x[lane >> 4][2 * k]) || is_zero(T.x[lane >> 4][2 * k + 1]));
        } else {
            zero = (lane >> 4) < t && (lane & 15) < len && is_zero(T.x[lane >> 4][lane & 15]);
        }
        const bool checked = __any_sync(0xffffffffu, zero) || len < kApplyK;
        if (!checked) {
#pragma unroll
            for (int k = 0; k < kApplyK; ++k) {
                const double xv = T.x[col][ES * k + part];
                if constexpr (CPLX) {
                    const double2 av = *reinterpret_cast<const double2*>(&T.a[k][2 * row]);
                    p = add_rn(p, mul_rn(xv, av.x));
                    q_ = add_rn(q_, mul_rn(xv, av.y));
                } else {
                    p = add_rn(p, mul_rn(xv, T.a[k][row]));
                }
            }
        } else {
            for (int k = 0; k < len; ++k) {
                const double xv = T.x[col][ES * k + part];
                const bool nz = !is_zero(xv);
                if constexpr (CPLX) {
                    const double2 av = *reinterpret_cast<const double2*>(&T.a[k][2 * row]);
                    p = add_rn(p, nz ? mul_rn(xv, av.x) : 0.0);
                    q_ = add_rn(q_, nz ? mul_rn(xv, av.y) : 0.0);
                } else {
                    p = add_rn(p, nz ? mul_rn(xv, T.a[k][row]) : 0.0);
                }
            }
        }
        __syncwarp();  // every lane is past this slot before it is refilled
    }
    cp_wait<0>();
    const int i = i0 + row;
    if constexpr (CPLX) {
        // (pr - qi, pi + qr): the other part's q
        const double other = __shfl_xor_sync(0xffffffffu, q_, 8);
        if (i < n && col < t) d.y[((size_t)col * d.ldy + i) * 2 + part] = part ? add_rn(p, other) : sub_rn(p, other);
    } else {
        if (i < n && col < t) d.y[(size_t)col * d.ldy + i] = p;
    }
}

// ---- Y := A^H X, X n x t, t <= 2 ---------------------------------------------
// PanelProduct.ApplyTranspose (PanelProduct.cs:44-55): y[j] = Dot(a[:, j], x) in
// ColumnOps.Dot's order; complex operator: pr = Ar^T xr, pi = Ar^T xi, qr = Ai^T xr,
// qi = Ai^T xi, then (pr + qi, pi - qr). One half-warp per output row j, lane L
// holding the partial sums of the terms = L mod 16; kDotAhead terms of a lane
// (256 bytes of the column each) are loaded before they are added.
constexpr int kDotAhead = 8;

template <bool CPLX>
__global__ void __launch_bounds__(128) power_apply_t_kernel(const __grid_constant__ Batch<PanelDesc> b) {
    using E = typename std::conditional<CPLX, double2, double>::type;
    constexpr int T = 2, NQ = CPLX ? 4 : 1, W = 4;
    const PanelDesc& d = batch_item(b, blockIdx.y);
    const int n = d.n, t = d.t;
    if ((int)blockIdx.x * 8 >= n) return;  // eight half-warps
    const int half = (int)(blockIdx.x * 8 + (threadIdx.x >> 4));
    const int L = threadIdx.x & 15, base = threadIdx.x & 16;
    // A half past the last row computes row 0 and drops it, so every shuffle
    // sees a converged warp.
    const bool active = half < n;
    const int j = active ? half : 0;
    const E* a = reinterpret_cast<const E*>(d.a) + (size_t)j * d.ld;
    const E* x0 = reinterpret_cast<const E*>(d.x);
    const E* x1 = x0 + (t > 1 ? (size_t)d.ldx : 0);  // one column: twice the same, the second dropped
    double acc[T][NQ] = {};
    auto term = [](double (&r)[NQ], E aij, E xc) {
        if constexpr (CPLX) {
            r[0] = add_rn(r[0], mul_rn(aij.x, xc.x));  // pr
            r[1] = add_rn(r[1], mul_rn(aij.x, xc.y));  // pi
            r[2] = add_rn(r[2], mul_rn(aij.y, xc.x));  // qr
            r[3] = add_rn(r[3], mul_rn(aij.y, xc.y));  // qi
        } else {
            r[0] = add_rn(r[0], mul_rn(aij, xc));
        }
    };
    const int n16 = (n / (4 * W)) * (4 * W);
    const int n4 = n >= W ? n16 + ((n - n16) / W) * W : 0;
    double res[T][NQ] = {};
    if (n >= W) {
        int i = L;
        for (; i + 16 * (kDotAhead - 1) < n16; i += 16 * kDotAhead) {
            E av[kDotAhead], u[kDotAhead], v[kDotAhead];
#pragma unroll
            for (int q = 0; q < kDotAhead; ++q) {
                av[q] = a[i + 16 * q];
                u[q] = x0[i + 16 * q];
                v[q] = x1[i + 16 * q];
            }
#pragma unroll
            for (int q = 0; q < kDotAhead; ++q) {
                term(acc[0], av[q], u[q]);
                term(acc[1], av[q], v[q]);
            }
        }
        for (; i < n16; i += 16) {
            const E av = a[i];
            term(acc[0], av, x0[i]);
            term(acc[1], av, x1[i]);
        }
        if (L < W)
            for (i = n16 + L; i < n4; i += W) {
                const E av = a[i];
                term(acc[0], av, x0[i]);
                term(acc[1], av, x1[i]);
            }
        __syncwarp();
#pragma unroll
        for (int c = 0; c < T; ++c)
#pragma unroll
            for (int q = 0; q < NQ; ++q) res[c][q] = netdot_combine(acc[c][q], L, base);
    }
    if (!active || L != 0) return;
    for (int i = n4; i < n; ++i) {  // scalar tail, in order
        const E av = a[i];
        term(res[0], av, x0[i]);
        term(res[1], av, x1[i]);
    }
#pragma unroll
    for (int c = 0; c < T; ++c) {
        if (c >= t) continue;
        if constexpr (CPLX)
            reinterpret_cast<double2*>(d.y)[(size_t)c * d.ldy + j] =
                make_double2(add_rn(res[c][0], res[c][3]), sub_rn(res[c][1], res[c][2]));
        else
            d.y[(size_t)c * d.ldy + j] = res[c][0];
    }
}

// ---- || abs(A)^p ||_1 ----------------------------------------------------------
// row := ones; p times row[j] := sum_i row[i] |a_ij|, sequential in i
// (OneNormOfAbsolutePower, MatrixExponential.cs:468-505); then the largest entry.
// All p passes of a matrix in one launch, by one cluster of CTAs (one CTA up to
// n = 128): every warp keeps 32 columns' sums, one per lane; the moduli arrive by
// cp.async in tiles of 32 rows, running ahead into the next pass; the new row
// vector goes to every CTA's shared memory as it is finished, and the cluster
// meets at its hardware barrier between passes. A launch per pass cost more than
// the pass: 27 launches of 28 us at n = 512, whose chains of 512 additions take
// 2 us.
constexpr int kChainRows = 32;
constexpr int kChainPitch = kChainRows + 2;  // doubles per staged column: 16-byte aligned, no bank conflicts
constexpr int kChainStages = 4;
constexpr int kChainMaxWarps = 4;
constexpr int kChainCluster = 8;

__device__ __forceinline__ void st_cluster(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

__global__ void __launch_bounds__(32 * kChainMaxWarps) abs_power_chain_kernel(const __grid_constant__ Batch<ChainDesc> b,
                                                                             int passes, int cs, int nmax) {
    extern __shared__ __align__(128) unsigned char chain_smem[];
    const int item = blockIdx.x / cs, rank = blockIdx.x % cs;
    const ChainDesc& d = batch_item(b, item);
    const int n = d.n, ld = d.ld;
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* ring = reinterpret_cast<double*>(chain_smem) + (size_t)warp * kChainStages * 32 * kChainPitch;
    double* vec = reinterpret_cast<double*>(chain_smem) + (size_t)warps * kChainStages * 32 * kChainPitch;  // [2][nv]
    const int nv = (nmax + 1) & ~1;
    const int tiles = (n + kChainRows - 1) / kChainRows;
    // This warp's groups of 32 columns: first, first + step, ...
    const int first = (rank * warps + warp) * 32, step = cs * warps * 32;
    const int groups = first < n ? (n - first + step - 1) / step : 0;
    // The staging pointer runs over (pass, group, tile). Rows past n are zeros
    // of the padded moduli (ld a multiple of 64).
    int sp = 0, sg = 0, sq = 0, slot_in = 0;
    auto stage = [&] {
        if (groups > 0 && sp < passes) {
            const int j0 = first + sg * step, ncol = min(32, n - j0);
            double* buf = ring + (size_t)slot_in * 32 * kChainPitch + (lane >> 4) * kChainPitch + (lane & 15) * 2;
            const double* src = d.mags + (size_t)(j0 + (lane >> 4)) * ld + sq * kChainRows + (lane & 15) * 2;
#pragma unroll
            for (int u = 0; u < 16; ++u)
                if (2 * u + (lane >> 4) < ncol) cp16(buf + u * 2 * kChainPitch, src + (size_t)(2 * u) * ld, true);
            if (++sq == tiles) {
                sq = 0;
                if (++sg == groups) {
                    sg = 0;
                    ++sp;
                }
            }
        }
        if (++slot_in == kChainStages) slot_in = 0;
        cp_commit();
    };
    for (int q = 0; q < kChainStages - 1; ++q) stage();
    for (int i = threadIdx.x; i < n; i += blockDim.x) vec[i] = 1.0;
    cluster_sync();  // every CTA of the cluster runs (and the ones are written)
    int slot = 0;
    for (int pass = 0; pass < passes; ++pass) {
        const double* row = vec + (pass & 1) * nv;
        double* next = vec + ((pass + 1) & 1) * nv;
        for (int g = 0; g < groups; ++g) {
            double sum = 0.0;
            for (int q = 0; q < tiles; ++q) {
                cp_wait<kChainStages - 2>();
                __syncwarp();
                stage();  // into the slot finished last trip
                const double* col = ring + (size_t)slot * 32 * kChainPitch + lane * kChainPitch;
                if (++slot == kChainStages) slot = 0;
                const double* rv = row + q * kChainRows;
                const int len = min(kChainRows, n - q * kChainRows);
                if (len == kChainRows) {
#pragma unroll
                    for (int r = 0; r < kChainRows; r += 2) {
                        const double2 m = *reinterpret_cast<const double2*>(col + r);
                        const double2 w = *reinterpret_cast<const double2*>(rv + r);
                        sum = add_rn(sum, mul_rn(w.x, m.x));
                        sum = add_rn(sum, mul_rn(w.y, m.y));
                    }
                } else {
#pragma unroll 4
                    for (int r = 0; r < len; ++r) sum = add_rn(sum, mul_rn(rv[r], col[r]));
                }
                __syncwarp();
            }
            const int j = first + g * step + lane;
            if (j < n) {
                if (pass + 1 < passes) {
                    for (int c = 0; c < cs; ++c) st_cluster(cluster_addr(next + j, c), sum);
                } else {
                    (passes & 1 ? d.next : d.row)[j] = sum;
                }
            }
        }
        cluster_sync();
    }
    cp_wait<0>();
}

template <class K>
void allow_smem(K kernel, std::atomic<bool>* done, int device, size_t bytes) {
    if (done[device].load(std::memory_order_acquire)) return;
    TNS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done[device].store(true, std::memory_order_release);
}

template <bool CPLX>
void launch_apply(Context& ctx, std::vector<PanelDesc>& v, int nmax, bool adjoint) {
    Batch<PanelDesc> b = make_batch(ctx, v);
    if (adjoint) {
        power_apply_t_kernel<CPLX><<<dim3((nmax + 7) / 8, b.count), 128, 0, ctx.stream>>>(b);
    } else {
        constexpr int smem = kApplyStages * (int)sizeof(ApplyTile<CPLX>);
        constexpr int rows = ApplyTile<CPLX>::ROWS;
        power_apply_kernel<CPLX><<<dim3((nmax + rows - 1) / rows, b.count), 32, smem, ctx.stream>>>(b);
    }
    TNS_CUDA(cudaGetLastError());
    ctx.kernel_launches++;
}

size_t chain_smem_bytes(int warps, int n) {
    return sizeof(double) * ((size_t)warps * kChainStages * 32 * kChainPitch + 2 * (size_t)round_up(n, 2));
}
constexpr size_t kChainMaxSmem = 220 * 1024;

}  // namespace

void narrow_products(Context& ctx, std::vector<PanelDesc>& v, bool cplx, bool adjoint) {
    int nmax = 0;
    for (auto& d : v) nmax = std::max(nmax, d.n);
    if (nmax == 0) return;
    if (cplx) launch_apply<true>(ctx, v, nmax, adjoint);
    else launch_apply<false>(ctx, v, nmax, adjoint);
}

bool abs_power_chains(Context& ctx, const std::vector<ChainDesc>& v, int passes) {
    int nmax = 0;
    for (auto& d : v) nmax = std::max(nmax, d.n);
    if (nmax == 0) return true;
    // Warps of 32 columns: four to a CTA, up to eight CTAs to a cluster.
    const int warps = std::min(kChainMaxWarps, (nmax + 31) / 32);
    const int cs = std::min(kChainCluster, (nmax + 32 * warps - 1) / (32 * warps));
    const size_t smem = chain_smem_bytes(warps, nmax);
    if (smem > kChainMaxSmem) return false;
    static std::atomic<bool> done[64];
    allow_smem(abs_power_chain_kernel, done, ctx.device, kChainMaxSmem);
    Batch<ChainDesc> b = make_batch(ctx, v);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(cs * v.size()));
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    TNS_CUDA(cudaLaunchKernelEx(&cfg, abs_power_chain_kernel, b, passes, cs, nmax));
    ctx.kernel_launches++;
    return true;
}

}  // namespace tns
