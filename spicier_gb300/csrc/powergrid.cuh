// Power-grid corner sweep on the GPU: Newton with restarted GMRES and Jacobi
// preconditioning, one CTA per instance.
//
// The algorithm is the one stated in oracle/powergrid.hpp (which cites the
// reference for each part): full-step Newton from x = 0, each linear solve by
// right-preconditioned GMRES(m) with Givens rotations; the Arnoldi vectors
// are orthogonalised by classical Gram-Schmidt applied twice (the oracle and
// the reference use modified Gram-Schmidt: same iterates in exact
// arithmetic, two block reductions per step instead of k + 1).  Layout of the
// FP64 kernel: thread t of the CTA owns rows t, t + T, t + 2T, ... of every
// vector (coalesced), the edge conductances and the Krylov basis live in the
// instance's global workspace (an FP64 basis does not fit on chip; for the FP32
// one see powergrid_mixed.cuh), the vector being multiplied lives in shared
// memory for the stencil's neighbour reads, and every dot product is a
// fixed-order block reduction (so a run is reproducible; the oracle's
// sequential sums round differently).
//
//   SP_PREC_FP64   the oracle's algorithm in FP64 (GMRES on A x_new = b);
//   SP_PREC_MIXED  FP32 Krylov: each Newton iteration solves A d = b - A x
//                  with the basis, the stencil and the projections in FP32
//                  to a relative 1e-3, the residual b - A x and the update in
//                  FP64; Newton runs until the reference's step test passes
//                  and max |KCL residual| <= resid_target (this is the FP64
//                  refinement of the FP32 solves).
#pragma once
#include "internal.h"
#include "rng.cuh"

namespace sp {

constexpr int kGridThreads = 512;
constexpr int kGridMaxRestart = 32;
constexpr int kGridRowsPerThread = 9;  // n <= 4608 unknowns

struct GridLaunch {
    sp_grid_config cfg;
    uint64_t seed, first, count;
    void* ws;          // per instance: ws + i * ws_stride bytes
    size_t ws_stride;  // bytes
    int max_smem;      // dynamic shared memory a block may have
    double* x;         // [count][n]
    int32_t* newton;
    int32_t* krylov;
    uint8_t* status;
    double* resid;
};

// Byte offsets inside one instance's workspace (n = rows * cols + 1).
struct GridWs {
    size_t gh, gv, diag, b, r, sink, vgs, sids, sgds, V, total;
};

__host__ __device__ inline size_t gws_align(size_t b) { return (b + 255) & ~size_t(255); }

__host__ __device__ inline GridWs grid_ws(const sp_grid_config& c, int vbytes) {
    const size_t R = c.rows, Cn = c.cols, n = R * Cn + 1, m = c.restart;
    GridWs w;
    size_t o = 0;
    w.gh = o; o += gws_align(8 * R * (Cn - 1));
    w.gv = o; o += gws_align(8 * (R - 1) * Cn);
    w.diag = o; o += gws_align(8 * n);
    w.b = o; o += gws_align(8 * n);
    w.r = o; o += gws_align(8 * n);
    w.sink = o; o += gws_align(4 * (size_t)c.num_sinks);
    w.vgs = o; o += gws_align(8 * (size_t)c.num_sinks);
    w.sids = o; o += gws_align(8 * (size_t)c.num_sinks);
    w.sgds = o; o += gws_align(8 * (size_t)c.num_sinks);
    w.V = o; o += gws_align((size_t)vbytes * n * (m + 1));
    w.total = o;
    return w;
}

// Dynamic shared memory of grid_kernel for Krylov element size `tb`.
__host__ __device__ inline size_t grid_smem_bytes(const sp_grid_config& c, int tb) {
    const size_t n = (size_t)c.rows * c.cols + 1;
    const size_t head = (3 * (size_t)tb * n + 15) & ~size_t(15);
    const size_t dense = 8 * ((size_t)kGridMaxRestart * (kGridMaxRestart + 1) + (kGridMaxRestart + 1) + 3 * kGridMaxRestart);
    return head + dense + (size_t)tb * 64 + 8 * 32 + (size_t)tb * ((kGridThreads / 32 + 1) * (kGridMaxRestart + 1));
}

#ifdef SP_KERNEL_NS
namespace SP_KERNEL_NS {

// Maximum over the first T threads (order-free).
template <int T = kGridThreads>
__device__ inline double block_max(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double m = 0.0;
    for (int w = 0; w < T / 32; ++w) m = fmax(m, red[w]);
    __syncthreads();
    return m;
}

// Fixed-order block sum over kGridThreads threads (warp tree, then warp 0).
template <class T>
__device__ inline T block_sum(T v, T* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();  // red[] free
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        T s = lane < kGridThreads / 32 ? red[lane] : T(0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[32] = s;
    }
    __syncthreads();
    return red[32];
}

// y = A z for the rows of this thread (z in shared memory), in the oracle's
// term order; T is the arithmetic type of the product.
template <class T>
__device__ inline T grid_apply_row(const sp_grid_config& c, const double* gh, const double* gv, const T* diag,
                                   const T* z, int p) {
    const int R = c.rows, Cn = c.cols, nn = R * Cn;
    if (p == nn) return z[0];
    const int r = p / Cn, j = p - r * Cn;
    T v = diag[p] * z[p];
    if (j > 0) v -= (T)gh[r * (Cn - 1) + j - 1] * z[p - 1];
    if (j < Cn - 1) v -= (T)gh[r * (Cn - 1) + j] * z[p + 1];
    if (r > 0) v -= (T)gv[(r - 1) * Cn + j] * z[p - Cn];
    if (r < R - 1) v -= (T)gv[r * Cn + j] * z[p + Cn];
    const int c1 = Cn - 1, c2 = (R - 1) * Cn, c3 = nn - 1;
    if (p == 0) {
        v -= (T)c.strap_g * z[c1];
        v -= (T)c.strap_g * z[c2];
        v -= (T)c.strap_g * z[c3];
        v += z[nn];
    } else if (p == c1 || p == c2 || p == c3) {
        v -= (T)c.strap_g * z[0];
    }
    return v;
}

// Rows (and sinks) of thread t start at t and are T apart; threads past the first T own none.
template <int T>
__device__ inline int grid_first(int none) {
    return threadIdx.x < T ? (int)threadIdx.x : none;
}

// Pointers into one instance's workspace.
struct GridPtrs {
    double *gh, *gv, *diag, *b, *r, *vgs, *sids, *sgds;
    int* sink;
    unsigned char* V;
};

__device__ inline GridPtrs grid_ptrs(const GridLaunch& L, const GridWs& W, uint32_t i) {
    unsigned char* base = (unsigned char*)L.ws + (size_t)i * L.ws_stride;
    GridPtrs g;
    g.gh = (double*)(base + W.gh);
    g.gv = (double*)(base + W.gv);
    g.diag = (double*)(base + W.diag);
    g.b = (double*)(base + W.b);
    g.r = (double*)(base + W.r);
    g.sink = (int*)(base + W.sink);
    g.vgs = (double*)(base + W.vgs);
    g.sids = (double*)(base + W.sids);
    g.sgds = (double*)(base + W.sgds);
    g.V = base + W.V;
    return g;
}

// The instance's draws, in the oracle's order (edges horizontal, vertical;
// sinks node, VGS), and x = 0.  Ends with a barrier.
template <int T>
__device__ inline void grid_draws(const GridLaunch& L, const GridPtrs& g, uint32_t inst, double* x) {
    const sp_grid_config& c = L.cfg;
    const int nn = c.rows * c.cols;
    const uint32_t layout = inst / 4, corner = inst % 4;
    const double scale = (corner & 1) ? c.r_scale_hi : c.r_scale_lo;
    unsigned hard = 0;
    const double lr = cr_log(c.r_hi / c.r_lo, &hard);
    const int nh = c.rows * (c.cols - 1), nv = (c.rows - 1) * c.cols;
    for (int e = grid_first<T>(nh + nv); e < nh + nv; e += T) {
        const double u = rng_uniform(L.seed, layout, (uint32_t)e);
        const double cond = 1.0 / (c.r_lo * cr_exp(u * lr, &hard) * scale);
        if (e < nh) g.gh[e] = cond;
        else g.gv[e - nh] = cond;
    }
    for (int s = grid_first<T>(c.num_sinks); s < c.num_sinks; s += T) {
        const uint32_t idx = (uint32_t)(nh + nv + 2 * s);
        g.sink[s] = (int)floor((double)nn * rng_uniform(L.seed, layout, idx));
        g.vgs[s] = c.vgs_lo + rng_uniform(L.seed, layout, idx + 1) * (c.vgs_hi - c.vgs_lo);
    }
    for (int p = grid_first<T>(nn + 1); p <= nn; p += T) x[p] = 0.0;
    __syncthreads();
}

__device__ inline double grid_vto(const sp_grid_config& c, uint32_t inst) {
    return (inst % 4 & 2) ? c.vto + c.vto_shift : c.vto - c.vto_shift;
}

// Diagonal and right-hand side of the system linearised at x.  Each node's
// sinks are added in sink order by the node's owner, which walks the whole
// list (one walker took 512 dependent round trips to memory per iteration).
// Ends without a barrier: rows of diag and b belong to their thread.
template <int T>
__device__ inline void grid_linearise(const sp_grid_config& c, const GridPtrs& g, double vto, double beta,
                                      const double* x) {
    const int nn = c.rows * c.cols, n = nn + 1, tid = threadIdx.x;
    for (int s = grid_first<T>(c.num_sinks); s < c.num_sinks; s += T) {
        const double vds = x[g.sink[s]], vg = g.vgs[s], vth = fabs(vto);
        double ids, gds;
        if (vg < vth) {
            ids = 0.0;
            gds = 1e-12;
        } else if (vds < vg - vth) {
            const double vov = vg - vth;
            ids = beta * (vov * vds - 0.5 * vds * vds) * (1.0 + c.lambda * vds);
            gds = fmax(beta * (vov - vds) * (1.0 + c.lambda * vds) + beta * (vov * vds - 0.5 * vds * vds) * c.lambda,
                       1e-12);
        } else {
            const double vov = vg - vth;
            ids = 0.5 * beta * vov * vov * (1.0 + c.lambda * vds);
            gds = fmax(0.5 * beta * vov * vov * c.lambda, 1e-12);
        }
        g.sids[s] = ids - gds * vds;
        g.sgds[s] = gds;
    }
    for (int p = grid_first<T>(n); p < n; p += T) {
        double d = 0.0;
        if (p < nn) {
            const int rr = p / c.cols, j = p - rr * c.cols;
            if (j > 0) d += g.gh[rr * (c.cols - 1) + j - 1];
            if (j < c.cols - 1) d += g.gh[rr * (c.cols - 1) + j];
            if (rr > 0) d += g.gv[(rr - 1) * c.cols + j];
            if (rr < c.rows - 1) d += g.gv[rr * c.cols + j];
            if (p == 0) d += 3.0 * c.strap_g;
            else if (p == c.cols - 1 || p == (c.rows - 1) * c.cols || p == nn - 1) d += c.strap_g;
        }
        g.diag[p] = d;
        g.b[p] = p < nn ? 0.0 : c.vdd;
    }
    __syncthreads();
    if (tid < T) {
#pragma unroll 4
        for (int s = 0; s < c.num_sinks; ++s) {
            const int p = g.sink[s];
            if ((p & (T - 1)) == tid) {
                g.diag[p] += g.sgds[s];
                g.b[p] -= g.sids[s];
            }
        }
    }
}

// KCL residual at the final iterate (FP64): the largest |A(x) x - b(x)| of the node rows.
template <int T>
__device__ inline double grid_residual(const sp_grid_config& c, const GridPtrs& g, double vto, double beta,
                                       const double* x, double* redd) {
    const int nn = c.rows * c.cols, tid = threadIdx.x;
    for (int s = grid_first<T>(c.num_sinks); s < c.num_sinks; s += T) {
        const double vds = x[g.sink[s]], vg = g.vgs[s], vth = fabs(vto);
        double ids;
        if (vg < vth) ids = 0.0;
        else if (vds < vg - vth) {
            const double vov = vg - vth;
            ids = beta * (vov * vds - 0.5 * vds * vds) * (1.0 + c.lambda * vds);
        } else {
            const double vov = vg - vth;
            ids = 0.5 * beta * vov * vov * (1.0 + c.lambda * vds);
        }
        g.sids[s] = ids;
    }
    for (int p = grid_first<T>(nn); p < nn; p += T) {
        const int rr = p / c.cols, j = p - rr * c.cols;
        double v = 0.0;  // currents leaving node p through the grid and straps
        if (j > 0) v += g.gh[rr * (c.cols - 1) + j - 1] * (x[p] - x[p - 1]);
        if (j < c.cols - 1) v += g.gh[rr * (c.cols - 1) + j] * (x[p] - x[p + 1]);
        if (rr > 0) v += g.gv[(rr - 1) * c.cols + j] * (x[p] - x[p - c.cols]);
        if (rr < c.rows - 1) v += g.gv[rr * c.cols + j] * (x[p] - x[p + c.cols]);
        if (p == 0) {
            v += c.strap_g * (x[0] - x[c.cols - 1]);
            v += c.strap_g * (x[0] - x[(c.rows - 1) * c.cols]);
            v += c.strap_g * (x[0] - x[nn - 1]);
            v += x[nn];
        } else if (p == c.cols - 1 || p == (c.rows - 1) * c.cols || p == nn - 1) {
            v += c.strap_g * (x[p] - x[0]);
        }
        g.r[p] = v;
    }
    __syncthreads();
    if (tid < T) {
#pragma unroll 4
        for (int s = 0; s < c.num_sinks; ++s) {
            const int p = g.sink[s];
            if ((p & (T - 1)) == tid) g.r[p] += g.sids[s];
        }
    }
    double mx = 0.0;
    for (int p = grid_first<T>(nn); p < nn; p += T) mx = fmax(mx, fabs(g.r[p]));
    return block_max<T>(mx, redd);
}

__global__ void __launch_bounds__(kGridThreads, 1) grid_kernel(GridLaunch L) {
    using T = double;
    extern __shared__ __align__(16) unsigned char gsm[];
    const sp_grid_config& c = L.cfg;
    const int n = c.rows * c.cols + 1, nn = n - 1, m = c.restart;
    const int tid = threadIdx.x;
    const uint32_t i = blockIdx.x;
    const uint32_t inst = (uint32_t)(L.first + i);
    const GridWs W = grid_ws(c, (int)sizeof(T));
    const GridPtrs g = grid_ptrs(L, W, i);
    double *gh = g.gh, *gv = g.gv, *diag = g.diag, *b = g.b, *r = g.r;
    T* V = (T*)g.V;
    // shared: z (the vector multiplied, T), Jacobi inverse in T, small dense parts
    T* zs = reinterpret_cast<T*>(gsm);
    T* inv = zs + n;
    T* dT = inv + n;  // diag in the Krylov type
    double* hmat = reinterpret_cast<double*>(gsm + ((3 * sizeof(T) * n + 15) & ~size_t(15)));
    double* gvec = hmat + kGridMaxRestart * (kGridMaxRestart + 1);
    double* cs = gvec + kGridMaxRestart + 1;
    double* sn = cs + kGridMaxRestart;
    double* yv = sn + kGridMaxRestart;
    T* red = reinterpret_cast<T*>(yv + kGridMaxRestart);
    double* redd = reinterpret_cast<double*>(red + 64);  // 32 doubles
    T* proj = reinterpret_cast<T*>(redd + 32);           // [warps][kGridMaxRestart + 1]
    T* hcol = proj + (kGridThreads / 32) * (kGridMaxRestart + 1);
    double* x = L.x + (size_t)i * n;

    grid_draws<kGridThreads>(L, g, inst, x);
    const double vto = grid_vto(c, inst);

    int newton_it = 0, krylov_total = 0;
    uint8_t status = SP_ST_FAILED;
    double resid = 0.0;
    const double beta = c.kp * 1.0 * c.w / c.l;  // level1.rs:68-70 (NF = 1)
    for (int it = 1; it <= c.max_newton; ++it) {
        grid_linearise<kGridThreads>(c, g, vto, beta, x);
        for (int p = tid; p < n; p += kGridThreads) {
            inv[p] = (T)(fabs(diag[p]) < 1e-30 ? 1.0 : 1.0 / diag[p]);
            dT[p] = (T)diag[p];
        }
        for (int p = tid; p < n; p += kGridThreads) r[p] = b[p];
        __syncthreads();
        // --- GMRES on A x_new = b
        // sol lives in b's storage after this point (b is no longer needed)
        double* sol = b;
        for (int p = tid; p < n; p += kGridThreads) sol[p] = 0.0;
        T rnorm2_local = 0;
        for (int p = tid; p < n; p += kGridThreads) rnorm2_local += (T)r[p] * (T)r[p];
        const double b_norm = sqrt((double)block_sum<T>(rnorm2_local, red));
        const double tol = c.krylov_tol;
        int total = 0;
        bool solved = b_norm < 1e-30;
        for (int cycle = 0; !solved && cycle < c.max_krylov; ++cycle) {
            // residual of the current solution, r - A sol
            __syncthreads();
            T loc = 0;
            for (int p = tid; p < n; p += kGridThreads) {
                const double rv = r[p] - grid_apply_row<double>(c, gh, gv, diag, sol, p);
                V[p] = (T)rv;
                loc += (T)rv * (T)rv;
            }
            const double r_norm = sqrt((double)block_sum<T>(loc, red));
            if (r_norm / b_norm < tol) {
                solved = true;
                break;
            }
            const T inv_r = (T)(1.0 / r_norm);
            for (int p = tid; p < n; p += kGridThreads) V[p] *= inv_r;
            if (tid <= m) gvec[tid] = 0.0;
            __syncthreads();
            if (tid == 0) gvec[0] = r_norm;
            int k = 0;
            while (k < m) {
                ++total;
                if (total > c.max_krylov) break;
                // z_k = M^-1 v_k into shared memory; w = A z_k
                for (int p = tid; p < n; p += kGridThreads) zs[p] = V[(size_t)k * n + p] * inv[p];
                __syncthreads();
                T w[kGridRowsPerThread];
#pragma unroll
                for (int q = 0; q < kGridRowsPerThread; ++q) {
                    const int p = tid + q * kGridThreads;
                    w[q] = p < n ? grid_apply_row<T>(c, gh, gv, dT, zs, p) : T(0);
                }
                // classical Gram-Schmidt, applied twice (CGS2): one block
                // reduction of all k+1 projections per pass instead of one per
                // basis vector; in exact arithmetic the same Hessenberg column
                // as modified Gram-Schmidt, and as well conditioned in practice
                for (int pass = 0; pass < 2; ++pass) {
                    // projections in chunks of 8 basis vectors: the chunk's loads
                    // are independent, so they overlap instead of one at a time
                    for (int j0 = 0; j0 <= k; j0 += 8) {
                        T acc[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            acc[u] = 0;
                            if (j0 + u <= k) {
                                const T* vj = V + (size_t)(j0 + u) * n;
#pragma unroll
                                for (int q = 0; q < kGridRowsPerThread; ++q) {
                                    const int p = tid + q * kGridThreads;
                                    if (p < n) acc[u] += vj[p] * w[q];
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            T v = acc[u];
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                            if ((tid & 31) == 0 && j0 + u <= k) proj[(tid >> 5) * (kGridMaxRestart + 1) + j0 + u] = v;
                        }
                    }
                    __syncthreads();
                    if (tid <= k) {
                        T hs = 0;
                        for (int w2 = 0; w2 < kGridThreads / 32; ++w2) hs += proj[w2 * (kGridMaxRestart + 1) + tid];
                        hcol[tid] = hs;
                        hmat[k * (kGridMaxRestart + 1) + tid] = pass == 0 ? (double)hs
                                                                          : hmat[k * (kGridMaxRestart + 1) + tid] + (double)hs;
                    }
                    __syncthreads();
                    for (int j0 = 0; j0 <= k; j0 += 8) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            if (j0 + u <= k) {
                                const T hij = hcol[j0 + u];
                                const T* vj = V + (size_t)(j0 + u) * n;
#pragma unroll
                                for (int q = 0; q < kGridRowsPerThread; ++q) {
                                    const int p = tid + q * kGridThreads;
                                    if (p < n) w[q] -= hij * vj[p];
                                }
                            }
                        }
                    }
                }
                T loc3 = 0;
#pragma unroll
                for (int q = 0; q < kGridRowsPerThread; ++q) loc3 += w[q] * w[q];
                const double w_norm = sqrt((double)block_sum<T>(loc3, red));
                if (w_norm < 1e-30) {
                    if (tid == 0) hmat[k * (kGridMaxRestart + 1) + k + 1] = w_norm;
                    __syncthreads();
                    ++k;
                    break;
                }
                const T inv_w = (T)(1.0 / w_norm);
#pragma unroll
                for (int q = 0; q < kGridRowsPerThread; ++q) {
                    const int p = tid + q * kGridThreads;
                    if (p < n) V[(size_t)(k + 1) * n + p] = w[q] * inv_w;
                }
                if (tid == 0) {
                    double* hk = hmat + k * (kGridMaxRestart + 1);
                    hk[k + 1] = w_norm;
                    for (int j = 0; j < k; ++j) {
                        const double temp = cs[j] * hk[j] + sn[j] * hk[j + 1];
                        hk[j + 1] = -sn[j] * hk[j] + cs[j] * hk[j + 1];
                        hk[j] = temp;
                    }
                    double cc = 1.0, ss = 0.0;
                    if (fabs(hk[k + 1]) >= 1e-30) {
                        const double rr2 = sqrt(hk[k] * hk[k] + hk[k + 1] * hk[k + 1]);
                        cc = hk[k] / rr2;
                        ss = hk[k + 1] / rr2;
                    }
                    cs[k] = cc;
                    sn[k] = ss;
                    hk[k] = cc * hk[k] + ss * hk[k + 1];
                    hk[k + 1] = 0.0;
                    const double tg = cc * gvec[k] + ss * gvec[k + 1];
                    gvec[k + 1] = -ss * gvec[k] + cc * gvec[k + 1];
                    gvec[k] = tg;
                    redd[0] = fabs(gvec[k + 1]) / b_norm;
                }
                __syncthreads();
                const double rel = redd[0];
                ++k;
                if (rel < tol) break;
            }
            // y from the triangular system; sol += M^-1 V y
            if (tid == 0)
                for (int a = k - 1; a >= 0; --a) {
                    double sum = gvec[a];
                    for (int j = a + 1; j < k; ++j) sum -= hmat[j * (kGridMaxRestart + 1) + a] * yv[j];
                    const double haa = hmat[a * (kGridMaxRestart + 1) + a];
                    yv[a] = fabs(haa) > 1e-30 ? sum / haa : 0.0;
                }
            __syncthreads();
            for (int p = tid; p < n; p += kGridThreads) {
                double s = sol[p];
                for (int a = 0; a < k; ++a) s += (double)(V[(size_t)a * n + p] * inv[p]) * yv[a];
                sol[p] = s;
            }
            __syncthreads();
            if (total >= c.max_krylov) break;
        }
        krylov_total += total;
        // --- Newton update and the reference's convergence test
        bool ok = true, fin = true;
        for (int p = tid; p < n; p += kGridThreads) {
            const double old = x[p];
            const double nw = sol[p];
            const double tl = c.v_reltol * fmax(fabs(nw), fabs(old)) + (p < nn ? c.v_abstol : c.i_abstol);
            ok = ok && fabs(nw - old) <= tl;
            fin = fin && isfinite(nw);
            x[p] = nw;
        }
        ok = __syncthreads_and(ok);
        fin = __syncthreads_and(fin);
        newton_it = it;
        if (!fin) {
            status = SP_ST_NONFINITE;
            break;
        }
        if (ok) {
            status = SP_ST_CONVERGED;
            break;
        }
    }
    resid = grid_residual<kGridThreads>(c, g, vto, beta, x, redd);
    if (tid == 0) {
        L.newton[i] = newton_it;
        L.krylov[i] = krylov_total;
        L.status[i] = status;
        L.resid[i] = resid;
    }
}

}  // namespace SP_KERNEL_NS
#endif  // SP_KERNEL_NS

}  // namespace sp
