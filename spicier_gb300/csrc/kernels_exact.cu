// Kernels that reproduce the reference's IEEE operation sequence.
// Compiled with --fmad=false: no a*b+c is fused, as in the Rust reference.
#define SP_KERNEL_NS kexact
#define SP_EXACT_UNIT
#include "internal.h"
#include <math_constants.h>

#include "rng.cuh"
#include "ladder.cuh"
#include "transient_fixed.cuh"
#define SP_AC_KERNELS
#include "ac.cuh"
#include "ac_sparse.cuh"

namespace sp {

// Persistent draw kernel: each block takes groups of 32 samples from a
// device counter (a static stride without one) and, per group,
//
//   draws     warp w draws the non-fixed slots drawn[w], drawn[w + 8], ...
//             of the 32 samples (one distribution per warp), then writes
//             its share of the fixed slots;
//   derives   after the block barrier, lane y derives the constants of
//             elements y, y + 8, ... of each sample (fixed slots read from
//             the circuit, drawn ones from the values just written).
//
// A Gaussian is about a thousand integer instructions plus a few FP64 ones
// (the products and the square root), so the kernel is bound by the integer
// ALU pipe; taking groups from a counter keeps every SM busy to the end,
// where a fixed grid of short blocks would leave its last partial wave.
constexpr int kDrawSamples = 32, kDrawLanes = 8;

__global__ void __launch_bounds__(kDrawSamples * kDrawLanes, 4) draw_kernel(DrawLaunch L) {
    pdl_wait();
    pdl_trigger();
    __shared__ unsigned int group_s;
    // linear warm start (x0_out set): weights lin[nout][nin], in_mean[nin],
    // out_mean[nout], then the group's centred inputs pin[nin][32]
    extern __shared__ float lsm[];
    const int nin = L.lin_nin, nout = L.lin_nout;
    float* lin_s = lsm;
    float* inm_s = lsm + nout * nin;
    float* outm_s = inm_s + nin;
    float* pin_s = outm_s + nout;
    const DevCircuit& c = L.c;
    const int lane = threadIdx.x, warp = threadIdx.y;
    const int tid = warp * kDrawSamples + lane;
    if (L.x0_out) {
        for (int i = tid; i < nout * nin; i += kDrawSamples * kDrawLanes) lin_s[i] = L.lin[i];
        for (int i = tid; i < nin; i += kDrawSamples * kDrawLanes) inm_s[i] = L.lin_io[i];
        for (int i = tid; i < nout; i += kDrawSamples * kDrawLanes) outm_s[i] = L.lin_io[2 * nin + i];
    }
    const uint64_t groups = (L.count + kDrawSamples - 1) / kDrawSamples;
    unsigned hard = 0;
    for (uint64_t it = 0;; ++it) {
        if (lane == 0 && warp == 0) group_s = L.next ? atomicAdd(L.next, 1u) : (unsigned)(blockIdx.x + it * gridDim.x);
        __syncthreads();
        const uint64_t g = L.next ? (uint64_t)group_s : blockIdx.x + it * gridDim.x;
        if (g >= groups) break;  // the same value in every thread of the block
        const uint64_t s = g * kDrawSamples + (uint64_t)lane;
        const bool live = s < L.count;
        const uint32_t sweep = (uint32_t)(L.first_index + s);
        if (live) {
            const double* row = L.table ? L.table + s * L.table_cols : nullptr;
            for (int d = warp; d < L.num_drawn; d += kDrawLanes) {
                const int k = L.drawn[d];
                const double v = draw_one(c.par[k], L.seed, sweep, row, &hard);
                L.params_soa[(size_t)k * L.count + s] = v;
                if (L.params_out) L.params_out[s * c.num_params + k] = v;
            }
            for (int k = warp; k < c.num_params; k += kDrawLanes) {
                const sp_param p = c.par[k];
                if (p.kind != SP_DRAW_FIXED) continue;
                L.params_soa[(size_t)k * L.count + s] = p.a;
                if (L.params_out) L.params_out[s * c.num_params + k] = p.a;
            }
        }
        __syncthreads();  // this group's parameter slots are written (group_s is read by all)
        auto P = [&](int slot) {
            const sp_param& p = c.par[slot];
            return p.kind == SP_DRAW_FIXED ? p.a : L.params_soa[(size_t)slot * L.count + s];
        };
        if (L.x0_out) {  // the group's centred warm-start inputs, input j by warp j % 8
            for (int j = warp; j < nin; j += kDrawLanes)
                pin_s[j * kDrawSamples + lane] = live ? __double2float_rn(P(L.lin_slots[j])) - inm_s[j] : 0.f;
            __syncthreads();
        }
        if (!live) continue;
        if (L.derive)
            for (int e = warp; e < c.num_elements; e += kDrawLanes) {
                const sp_element el = c.el[e];
                double* out = L.derived_soa + (size_t)c.doff[e] * L.count + s;
                const size_t st = L.count;
                derive_element(el, P, [&](int k, double v) { out[k * st] = v; });
            }
        // linear warm start: lane y evaluates unknowns y, y + 8, ... in FP32 (as
        // the network kernels' linear term), inputs and weights from shared memory
        if (L.x0_out)
            for (int k = warp; k < nout; k += kDrawLanes) {
                float x = outm_s[k];
                for (int j = 0; j < nin; ++j) x = fmaf(lin_s[k * nin + j], pin_s[j * kDrawSamples + lane], x);
                L.x0_out[s * nout + k] = (double)x;
            }
    }
    if (hard && L.hard) atomicAdd(L.hard, hard);
}

// The draws alone, as work items of one warp each: item i is drawn slot
// drawn[i % num_drawn] of the 32-sample group i / num_drawn, taken from a
// device counter by the warp's lane 0.  Used when nothing in this kernel
// consumes a group's parameters together (no derived constants, no warm
// start, no row-major copy), so no block barrier is needed and every warp
// stays busy to the end, where whole groups per block spread a group's drawn
// slots unevenly over the 8 warps (17 slots: one warp draws three, the others
// two, and the block waits for it).  Fixed slots are not written (their
// consumers read them from the circuit).
__global__ void __launch_bounds__(kDrawSamples * kDrawLanes, 4) draw_items_kernel(DrawLaunch L) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const DevCircuit& c = L.c;
    const uint64_t groups = (L.count + kDrawSamples - 1) / kDrawSamples;
    const uint64_t items = groups * (uint64_t)L.num_drawn;
    unsigned hard = 0;
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(L.next_items, 1ULL);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= items) break;
        const uint64_t g = item / (uint64_t)L.num_drawn;
        const int k = L.drawn[(int)(item - g * (uint64_t)L.num_drawn)];
        const uint64_t s = g * kDrawSamples + (uint64_t)lane;
        if (s >= L.count) continue;
        const double* row = L.table ? L.table + s * L.table_cols : nullptr;
        L.params_soa[(size_t)k * L.count + s] = draw_one(c.par[k], L.seed, (uint32_t)(L.first_index + s), row, &hard);
    }
    if (hard && L.hard) atomicAdd(L.hard, hard);
}

// The draws of a sweep whose only consumer rounds them to FP32 (the
// double-float Newton kernel): FP32 values, Gaussians without the full draw
// where that decides the rounding (gauss_f32).  The work is even: a row of
// blocks per drawn slot, whose warps take 32-sample groups by a fixed stride.
__device__ __noinline__ static float draw_f32_full(const sp_param& p, uint64_t seed, uint32_t sweep, const double* row) {
    return __double2float_rn(draw_one(p, seed, sweep, row, nullptr));
}

__global__ void __launch_bounds__(256, 4) draw_f32_kernel(DrawLaunch L) {
    pdl_wait();
    pdl_trigger();
    const uint32_t lane = threadIdx.x & 31, groups = (uint32_t)((L.count + 31) / 32), warps = gridDim.x * 8;
    for (int slot = blockIdx.y; slot < L.num_drawn; slot += gridDim.y) {
        const int k = L.drawn[slot];
        const sp_param p = L.c.par[k];
        const uint64_t pk1 = (uint64_t)(p.rng_index * 2u) * 0x5851f42d4c957f2dULL;
        const uint64_t pk2 = (uint64_t)(p.rng_index * 2u + 1u) * 0x5851f42d4c957f2dULL;
        const float4 ms = L.gauss32[k];
        float* out = L.params32 + (size_t)k * L.count;
        for (uint32_t g = blockIdx.x * 8 + threadIdx.x / 32; g < groups; g += warps) {
            const uint64_t s = (uint64_t)g * 32 + lane;
            if (s >= L.count) continue;
            const uint32_t sweep = (uint32_t)(L.first_index + s);
            float v = 0.f;
            bool done = false;
            if (p.kind == SP_DRAW_GAUSS) done = gauss_f32(L.seed ^ (uint64_t)sweep * 0x517cc1b727220a95ULL, pk1, pk2, ms, &v);
            if (!done) v = draw_f32_full(L.c.par[k], L.seed, sweep, L.table ? L.table + s * L.table_cols : nullptr);
            out[s] = v;
        }
    }
}

cudaError_t launch_draw(const DrawLaunch& L, cudaStream_t st) {
    if (L.count == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    const uint64_t groups = (L.count + kDrawSamples - 1) / kDrawSamples;
    if (L.params32) {
        if (L.num_drawn == 0) return cudaSuccess;
        // one row of blocks per slot, about eight blocks per SM in all, and as few
        // warps per row as take the same number of groups each
        const uint64_t row = std::max<uint64_t>(1, ((uint64_t)sms * 8 + L.num_drawn - 1) / L.num_drawn);
        const uint64_t each = (groups + row * 8 - 1) / (row * 8);
        const uint64_t gx = (groups + each * 8 - 1) / (each * 8);
        return launch_chained(draw_f32_kernel, dim3((unsigned)gx, (unsigned)std::min(L.num_drawn, 65535)), dim3(256), 0, st, L);
    }
    if (L.next_items && !L.derive && !L.x0_out && !L.params_out) {
        if (L.num_drawn == 0) return cudaSuccess;
        const uint64_t warps = groups * (uint64_t)L.num_drawn;
        const uint64_t grid = std::min<uint64_t>((warps + kDrawLanes - 1) / kDrawLanes, (uint64_t)sms * 4);
        return launch_chained(draw_items_kernel, dim3((unsigned)grid), dim3(kDrawSamples * kDrawLanes), 0, st, L);
    }
    // resident blocks (four per SM at 64 registers); without a counter one block per group
    const uint64_t grid = L.next ? std::min<uint64_t>(groups, (uint64_t)sms * 4) : groups;
    const size_t smem = L.x0_out ? sizeof(float) * ((size_t)L.lin_nout * L.lin_nin + L.lin_nin + L.lin_nout +
                                                    (size_t)L.lin_nin * kDrawSamples)
                                 : 0;
    return launch_chained(draw_kernel, dim3((unsigned)grid), dim3(kDrawSamples, kDrawLanes), smem, st, L);
}

// Batched Bsim3Mosfet::evaluate (one thread per device): the per-sample
// constants from the device's card, then the evaluation at its bias.
__global__ void bsim3_eval_kernel(int pmos, const double* __restrict__ card, const double* __restrict__ bias,
                                  uint64_t count, double* __restrict__ out, uint8_t* __restrict__ region) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const double* c = card + i * SP_B3_CARD;
    double k[B3C_COUNT];
    bsim3_constants([&](int j) { return c[j]; }, [&](int j, double v) { k[j] = v; });
    const Bsim3Out r = bsim3_eval(pmos != 0, [&](int j) { return k[j]; }, bias[3 * i], bias[3 * i + 1], bias[3 * i + 2]);
    double* o = out + 6 * i;
    o[0] = r.ids;
    o[1] = r.gds;
    o[2] = r.gm;
    o[3] = r.gmbs;
    o[4] = r.vth;
    o[5] = r.vdsat;
    if (region) region[i] = (uint8_t)r.region;
}

cudaError_t launch_bsim3_eval(int pmos, const double* card, const double* bias, uint64_t count, double* out,
                              uint8_t* region, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    const int block = 128;
    bsim3_eval_kernel<<<(unsigned)((count + block - 1) / block), block, 0, st>>>(pmos, card, bias, count, out,
                                                                                region);
    return cudaGetLastError();
}

__global__ void rng_fill_kernel(int kind, uint64_t seed, uint64_t first, uint32_t param, uint64_t count,
                                double* out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t s = (uint32_t)(first + i);
    unsigned hard = 0;
    switch (kind) {
        case 0: out[i] = rng_uniform(seed, s, param); break;
        case 1: out[i] = rng_gaussian(seed, s, param, &hard); break;
        case 2: out[i] = (double)rng_uniform_f32(seed, s, param); break;
        default: out[i] = (double)rng_gaussian_f32(seed, s, param); break;
    }
}

cudaError_t launch_rng_fill(int kind, uint64_t seed, uint64_t first, uint32_t param, uint64_t count,
                            double* out, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    const int block = 256;
    rng_fill_kernel<<<(unsigned)((count + block - 1) / block), block, 0, st>>>(kind, seed, first, param,
                                                                              count, out);
    return cudaGetLastError();
}

cudaError_t launch_newton_exact(const NewtonLaunch& L, bool fallback, int grid, int block, size_t smem,
                                cudaStream_t st) {
    if (fallback) return launch_chained(SP_KERNEL_NS::newton_fallback_kernel<SP_PREC_FP64>, dim3(grid), dim3(block), smem, st, L);
    return launch_chained(SP_KERNEL_NS::newton_primary_kernel<SP_PREC_FP64>, dim3(grid), dim3(block), smem, st, L);
}

// BatchedLuSolver::solve_batch in FP64 with the reference's LU
// (CpuBatchedSolver, solver.rs:326-384): one thread per system, column-major
// input copied into interleaved shared memory; singular -> zero solution.
__global__ void lu_batch_fp64_kernel(const double* __restrict__ mats, const double* __restrict__ rhs,
                                     int n, uint64_t batch, double* __restrict__ sol,
                                     uint8_t* __restrict__ sing) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= batch) return;
    double* base = reinterpret_cast<double*>(smem);
    Il<double> A{base + threadIdx.x, (int)blockDim.x};
    Il<double> b{base + (size_t)n * n * blockDim.x + threadIdx.x, (int)blockDim.x};
    const double* m = mats + s * n * n;
    for (int i = 0; i < n * n; ++i) A[i] = m[i];
    for (int i = 0; i < n; ++i) b[i] = rhs[s * n + i];
    bool ok = lu_solve_fp64(n, A, b);
    for (int i = 0; i < n; ++i) sol[s * n + i] = ok ? b[i] : 0.0;
    sing[s] = ok ? 0 : 1;
}

cudaError_t launch_lu_batch_exact(const double* mats, const double* rhs, int n, uint64_t batch,
                                  double* sol, uint8_t* sing, cudaStream_t st) {
    if (batch == 0) return cudaSuccess;
    size_t per = (size_t)(n * n + n) * 8;
    int block = 128;
    while (block > 32 && per * block > 110 * 1024) block -= 32;
    size_t smem = per * block;
    lu_batch_fp64_kernel<<<(unsigned)((batch + block - 1) / block), block, smem, st>>>(mats, rhs, n, batch,
                                                                                     sol, sing);
    return cudaGetLastError();
}

// The same solve with one CTA per system.  Each step's pivot search (warp 0:
// first index of the largest |a|, NaN never chosen, the diagonal kept when it
// is NaN), row swap, scaling and rank-1 update apply to every element the
// operations of lu_solve_fp64 in the same order, only spread over threads, so
// the solution is bit-identical.  The right-hand side is column n of A: the
// update of that column is the forward substitution, so L needs no row swaps
// and is not read again.  A lives in shared memory when it fits, else in a
// per-CTA slice of global memory (work).
//
// Bound: the FP64 pipe, two lanes per clock and SM, whatever the number of
// active lanes; so nothing but the update's multiply and subtract runs on it.
// The trailing block's elements are dealt to full warps in column-major order
// (a warp that took rows of one column would idle on average a third of its
// lanes), the pivot search compares bit patterns, and the divisions, one per
// column and one per back-substitution step, run once per system on the
// integer pipe.  Warp 0 updates column i + 1 first and searches it while the
// other warps take the rest of the block in chunks.  65,535 systems of n = 50:
// 13.9 ms, 1.5 times the pipe's time for the multiplies and subtracts (29.1 ms
// with rows of a column per warp, the reciprocal in every warp and FP64
// compares); 2,000 of n = 100: 3.5 ms (5.0).  The multiply on the integer pipe
// beside the pipe's subtract measured slower (2.0 times at n = 50).
constexpr int kLuChunk = 4;  // elements per lane of one chunk

template <bool IN_WORK>
__global__ void __launch_bounds__(512) lu_batch_cta_kernel(const double* __restrict__ mats,
                                                           const double* __restrict__ rhs, int n, uint64_t batch,
                                                           double* __restrict__ sol, uint8_t* __restrict__ sing,
                                                           double* __restrict__ work) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_piv, s_bad;
    __shared__ double s_inv;
    __shared__ int s_next[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t nn = (size_t)n * n;
    double* A = IN_WORK ? work + (size_t)blockIdx.x * (nn + n) : reinterpret_cast<double*>(smem);
    // warp 0: pivot of column i into s_piv, 1 / pivot into s_inv, a zero pivot into s_bad
    auto find_pivot = [&](int i) {
        const double* col = A + (size_t)i * n;
        const uint64_t inf = 0x7FF0000000000000ULL;
        int piv = i;
        if ((cr::dbits(col[i]) << 1) <= (inf << 1)) {
            uint64_t best = 0;
            int bi = i;
            for (int r = i + lane; r < n; r += 32) {
                const uint64_t v = cr::dbits(col[r]) & ~(1ULL << 63);
                if (v > best && v <= inf) best = v, bi = r;
            }
            const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
            const bool top = (unsigned)(best >> 32) == hi;
            const unsigned lo = __reduce_max_sync(0xffffffffu, top ? (unsigned)best : 0u);
            piv = (int)__reduce_min_sync(0xffffffffu, top && (unsigned)best == lo ? (unsigned)bi : 0x7fffffffu);
            // a column of zeros: every lane holds best = 0 and lane 0's index is i
        }
        const double diag = col[piv];
        const bool zero = (cr::dbits(diag) << 1) == 0;
        const double inv = zero ? 0.0 : div_int(1.0, diag);
        if (lane == 0) {
            s_piv = piv;
            s_inv = inv;
            if (zero) s_bad = 1;
        }
    };
    for (uint64_t s = blockIdx.x; s < batch; s += gridDim.x) {
        const double* m = mats + s * nn;
        for (size_t k = tid; k < nn; k += blockDim.x) A[k] = m[k];
        for (int k = tid; k < n; k += blockDim.x) A[nn + k] = rhs[s * n + k];
        if (tid == 0) s_bad = 0, s_next[0] = s_next[1] = 0;
        __syncthreads();
        if (wid == 0) find_pivot(0);
        __syncthreads();
        for (int i = 0; i < n && !s_bad; ++i) {
            // swap rows i and piv in columns i.. n, scale column i below the diagonal
            const int piv = s_piv;
            const double inv = s_inv;
            double* col = A + (size_t)i * n;
            if (piv != i)
                for (int c = i + 1 + tid; c <= n; c += blockDim.x) {
                    double* cc = A + (size_t)c * n;
                    const double t = cc[i];
                    cc[i] = cc[piv];
                    cc[piv] = t;
                }
            const double cii = col[i], cpi = col[piv];
            __syncthreads();  // every thread has read the column's two entries
            for (int r = i + 1 + tid; r < n; r += blockDim.x) col[r] = (r == piv ? cii : col[r]) * inv;
            if (tid == 0) col[i] = cpi, s_next[(i + 1) & 1] = 0;
            __syncthreads();
            const int rows = n - 1 - i;
            if (rows == 0) break;
            const double* l = col + i + 1;
            if (wid == 0) {  // column i + 1, then its pivot
                double* cc = A + (size_t)(i + 1) * n + i;
                const double p = cc[0];
                for (int r = lane; r < rows; r += 32) cc[1 + r] = -p * l[r] + cc[1 + r];
                __syncwarp();
                find_pivot(i + 1);
            }
            // columns i + 2 .. n, element e of the block at row e % rows, column e / rows
            const int total = rows * rows;
            const int q32 = 32 / rows, r32 = 32 - q32 * rows;
            double* blk = A + (size_t)(i + 2) * n + i;
            while (true) {
                int e0 = 0;
                if (lane == 0) e0 = atomicAdd(&s_next[i & 1], 32 * kLuChunk);
                e0 = __shfl_sync(0xffffffffu, e0, 0);
                if (e0 >= total) break;
                int e = e0 + lane, c = e / rows, r = e - c * rows;
                double a[kLuChunk], p[kLuChunk], f[kLuChunk];
                int at[kLuChunk];  // the element's index in blk, -1 past the end
#pragma unroll
                for (int u = 0; u < kLuChunk; ++u) {
                    const bool live = e + 32 * u < total;
                    const int rr = live ? r : 0, k = (live ? c : 0) * n;
                    at[u] = live ? k + 1 + rr : -1;
                    a[u] = blk[k + 1 + rr];
                    p[u] = blk[k];
                    f[u] = l[rr];
                    r += r32;
                    c += q32;
                    if (r >= rows) r -= rows, ++c;
                }
#pragma unroll
                for (int u = 0; u < kLuChunk; ++u)
                    if (at[u] >= 0) blk[at[u]] = -p[u] * f[u] + a[u];
            }
            __syncthreads();
        }
        const bool bad = s_bad != 0;
        double* b = A + nn;
        if (wid == 0 && !bad) {  // back substitution (warp-synchronous); the diagonal is nonzero
            for (int i = n - 1; i >= 0; --i) {
                const double* col = A + (size_t)i * n;
                const double coeff = div_int(b[i], col[i]);
                __syncwarp();
                if (lane == 0) b[i] = coeff;
                for (int r = lane; r < i; r += 32) b[r] = -coeff * col[r] + b[r];
                __syncwarp();
            }
        }
        __syncthreads();
        for (int k = tid; k < n; k += blockDim.x) sol[s * n + k] = bad ? 0.0 : b[k];
        if (tid == 0) sing[s] = bad ? 1 : 0;
        __syncthreads();  // before the next system overwrites A and b
    }
}

size_t lu_batch_cta_smem(int n) { return ((size_t)n * n + n) * 8; }

cudaError_t launch_lu_batch_cta(const double* mats, const double* rhs, int n, uint64_t batch, double* sol,
                                uint8_t* sing, double* work, int grid, cudaStream_t st) {
    if (batch == 0) return cudaSuccess;
    const size_t smem = work ? 0 : lu_batch_cta_smem(n);
    // threads per system: enough to spread a step's (n - i)^2 elements, few
    // enough that its two barriers stay cheap.  Measured, ms for one batch per
    // n at 32 / 64 / 128 / 256 / 512 threads: n = 20 (65,535 systems) 1.70 /
    // 1.88 / 2.5 / - / -; n = 50 (16,500) 4.9 / 4.2 / 3.5 / 4.5 / -; n = 72
    // (5,858) 7.1 / 4.5 / 4.1 / 3.6 / -; n = 100 (2,500) - / 8.8 / 5.6 / 4.9 / 4.4
    const int block = n <= 22 ? 32 : n <= 40 ? 64 : n <= 64 ? 128 : n <= 88 ? 256 : 512;
    if (work)
        lu_batch_cta_kernel<true><<<grid, block, 0, st>>>(mats, rhs, n, batch, sol, sing, work);
    else
        lu_batch_cta_kernel<false><<<grid, block, smem, st>>>(mats, rhs, n, batch, sol, sing, work);
    return cudaGetLastError();
}

cudaError_t launch_ac(const AcLaunch& L, int grid, int block, size_t smem, int sparse_grid, int sparse_block,
                      cudaStream_t st) {
    if (L.cap) {  // else every sample is marked for the dense kernel
        int vblock = 128;  // n^2 doubles of shared memory per sample
        const size_t per = 8 * (size_t)L.c.n * L.c.n;
        while (vblock > 32 && (per * vblock > 110 * 1024 || L.count / vblock < 304)) vblock >>= 1;
        ac_values_kernel<<<(unsigned)((L.count + vblock - 1) / vblock), vblock, per * vblock, st>>>(L);
        ac_sparse_kernel<<<sparse_grid, sparse_block, ac_sparse_warp_bytes(L.c.n, L.cap) * (sparse_block / 32), st>>>(L);
    }
    ac_kernel<<<grid, block, smem, st>>>(L);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ac_status_kernel<<<(unsigned)((L.count + 255) / 256), 256, 0, st>>>(L.count, L.dc_status, L.singular,
                                                                       const_cast<uint8_t*>(L.dc_status));
    return cudaGetLastError();
}

cudaError_t launch_ladder_exact(const LadderLaunch& L, int grid, int threads, size_t smem, cudaStream_t st) {
    if (L.ws)
        SP_KERNEL_NS::ladder_kernel<SP_PREC_FP64_EXACT, true><<<grid, threads, smem, st>>>(L);
    else
        SP_KERNEL_NS::ladder_kernel<SP_PREC_FP64_EXACT, false><<<grid, threads, smem, st>>>(L);
    return cudaGetLastError();
}

cudaError_t launch_transient_exact(const TransientLaunch& L, int block, size_t smem, cudaStream_t st) {
    const unsigned grid = (unsigned)((L.count + block - 1) / block);
    SP_KERNEL_NS::transient_fixed_kernel<<<grid, block, smem, st>>>(L);
    return cudaGetLastError();
}

cudaError_t prepare_exact_kernels(int max_smem) {
    const void* fns[] = {(const void*)SP_KERNEL_NS::newton_primary_kernel<SP_PREC_FP64>,
                         (const void*)SP_KERNEL_NS::newton_fallback_kernel<SP_PREC_FP64>,
                         (const void*)SP_KERNEL_NS::transient_fixed_kernel,
                         (const void*)SP_KERNEL_NS::ladder_kernel<SP_PREC_FP64_EXACT, false>,
                         (const void*)SP_KERNEL_NS::ladder_kernel<SP_PREC_FP64_EXACT, true>, (const void*)ac_kernel, (const void*)ac_values_kernel,
                         (const void*)ac_sparse_kernel,
                         (const void*)lu_batch_fp64_kernel, (const void*)lu_batch_cta_kernel<false>};
    for (const void* f : fns) {
        cudaError_t e = allow_dynamic_smem(f, max_smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace sp
