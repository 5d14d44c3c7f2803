// Batched nonlinear transient of RC-diode ladders on the GPU.
//
// One CTA integrates one ladder from t = 0 to tstop; CTAs take ladders from a
// work counter in order of decreasing size (the longest first), so a single
// persistent launch covers instances of 10 to 514 unknowns.  Thread t owns
// sections k = 1 + t + T j: it draws their R and C, keeps their capacitor
// states, evaluates their diodes and assembles their rows; the tridiagonal
// solve of each Newton iteration is warp 0's, and the step controller's
// scalars are thread 0's.  The algorithm (step, controller, Newton per stage)
// is the one stated in oracle/transient.hpp, which cites the reference for
// every piece.
//
// What bounds it: the FP64 pipe (two lanes per clock and SM, about 20 FP64
// operations per section and Newton iteration) once several ladders share an
// SM, and the serial chain of the longest ladder when few do.  A ladder's
// arrays therefore live in shared memory (about 90 bytes a section, four
// ladders of 512 sections per SM; FP64 120 bytes, three), the per-section work is spread over the
// CTA, and the chain inside an iteration is kept to the elimination's
// dependent divisions.  One warp per ladder with its arrays in L2, the
// partition's 64-bit index divisions, a branch per division and bank conflicts
// in the chain took 44 us per Newton iteration of a 512-section ladder; the
// mixed iteration now takes 11.5 us alone on an SM: assembly 2.7 us (FP64
// pipe), elimination 6.1, update 1.8, and a step's scalars 4.5 us per step.
// 512 ladders of up to 512 sections: 238 -> 69 ms; 200 of them in FP64: 556 -> 304;
// 4,096 of them, mixed: 352 -> 138 ms.
//
// Precisions:
//   SP_PREC_FP64_EXACT  the oracle's operation sequence (full-step Newton,
//                       divisions, sequential elimination by one thread);
//                       with the portable transcendentals it is bit-identical
//                       to the oracle in its "cr" mode;
//   SP_PREC_FP64        the same with FMA contraction and the warp-parallel
//                       elimination;
//   SP_PREC_MIXED       correction form: FP64 KCL residual of the linearised
//                       stage (diode current linearised at the limited
//                       voltage, as the full-step form), FP32 Jacobian and
//                       FP32 elimination, FP64 update and convergence test.
#pragma once
#include <type_traits>

#include "internal.h"
#include "rng.cuh"
#include "fpconv.cuh"
#include "fpdiv.cuh"

namespace sp {

// Per-section FP64 arrays of one instance: section conductance and
// capacitance, the accepted state (node voltage and capacitor current), the
// stage's iterate, and the companion conductance and current.
enum LadderArray { LA_G, LA_C, LA_X, LA_IP, LA_XS, LA_GEQ, LA_IEQ, LA_COUNT };
// Solver arrays (FP32 in the mixed mode): diagonal, right-hand side, the two
// spikes, the negated sub-diagonal and the stage's constant part of the diagonal.
enum LadderSolve { LS_B, LS_D, LS_L, LS_R, LS_NG, LS_J, LS_COUNT };

// Elements of one solver array.  The elimination reads one row per lane and
// block, so the rows are stored [row in block][block] with 33 columns: lanes
// at the same row of 32 blocks, and threads at 32 consecutive rows of one
// block, touch 32 banks.  The exact mode keeps the rows in order.
__host__ __device__ inline int ladder_solve_len(int max_sections, int prec) {
    if (prec == SP_PREC_FP64_EXACT) return max_sections + 2;
    const int rows = (max_sections + 31) / 32 + 1;
    return 33 * (rows > 3 ? rows : 3);
}
// The longest ladder a precision takes: its solver arrays fit shared memory.
__host__ __device__ inline int ladder_max_sections(int prec) { return prec == SP_PREC_MIXED ? 3582 : 1790; }

constexpr int kLadderCtl = 16 + 2 * 8;  // doubles: step scalars, per-warp maxima (at most 8 warps)
constexpr int kLadderBlk = 32 * 12;     // solver values: the elimination's blocks (first, so 16-byte aligned)

// Dynamic shared memory of one CTA; ws: the FP64 arrays are in the global workspace.
__host__ __device__ inline size_t ladder_smem(int max_sections, int prec, bool ws) {
    const size_t S = (size_t)max_sections + 2, e = prec == SP_PREC_MIXED ? 4 : 8;
    size_t b = 8 * (size_t)kLadderCtl + e * kLadderBlk + (ws ? 0 : 8 * (size_t)LA_COUNT * S);
    b += e * ((size_t)LS_COUNT * ladder_solve_len(max_sections, prec) + 64);
    return ((b + 7) & ~size_t(7)) + 4 * S;
}

// Threads per ladder: enough that a thread owns a few sections, since the
// elimination between two block barriers is one warp's in any case.  512 /
// 4,096 ladders of up to 512 sections, mixed: 90 / 161 ms at 64 threads,
// 78 / 138 at 128, 76 / 195 at 256 (barriers, with the SM full).
__host__ __device__ inline int ladder_threads(int max_sections) {
    return max_sections <= 48 ? 32 : max_sections <= 160 ? 64 : 128;
}

struct LadderLaunch {
    sp_ladder_config cfg;
    uint64_t seed, first, count;
    const uint32_t* order;  // [count] instance order (largest first)
    unsigned int* next;     // work counter (zero before the launch)
    double* ws;             // [grid][LA_COUNT][max_sections + 2], or nullptr: shared memory
    double* x_final;        // [count][max_sections + 2]
    int32_t* n;
    int32_t* accepted;
    int32_t* rejected;
    int32_t* iters;
    uint8_t* status;
    double* probe;          // [count][num_probe] or nullptr
    double* steps;          // [count][max_rec] accepted step sizes, or nullptr
    int max_rec;            // steps recorded per instance (the first max_rec)
};

__host__ __device__ inline int ladder_sections(const sp_ladder_config& c, uint64_t seed, uint32_t inst) {
    const double span = (double)(c.max_sections - c.min_sections + 1);
    return c.min_sections + (int)floor(span * rng_uniform(seed, inst, 0));
}

// x mod per for x >= 0, per > 0: exact like fmod, from a quotient that is at
// most one off (x - k per is representable, and the fused product is exact).
__device__ inline double ladder_mod(double x, double per, double inv_per) {
    if (x < per) return x;
    const double k = floor(x * inv_per);
    if (!(k < 0x1p50)) return fmod(x, per);
    const double r = fma(-k, per, x);
    return r < 0.0 ? fma(-(k - 1.0), per, x) : r >= per ? fma(-(k + 1.0), per, x) : r;
}

__device__ inline double ladder_pulse(const sp_pulse& p, double t, double inv_per) {
    if (t < p.td) return p.v1;
    const double t_rel = p.per > 0.0 ? ladder_mod(t - p.td, p.per, inv_per) : t - p.td;
    if (t_rel < p.tr) return p.v1 + (p.v2 - p.v1) * t_rel / p.tr;
    if (t_rel < p.tr + p.pw) return p.v2;
    if (t_rel < p.tr + p.pw + p.tf) return p.v2 - (p.v2 - p.v1) * (t_rel - p.tr - p.pw) / p.tf;
    return p.v1;
}

#ifdef SP_KERNEL_NS
namespace SP_KERNEL_NS {

// Warp-parallel solve of the chain's tridiagonal system (rows 1..N, sub- and
// super-diagonal -g, diagonal B, right-hand side D; diagonally dominant, so
// no pivoting): the partition method.  The rows are split into P contiguous
// blocks (P = min(32, N/2), one per lane, `len` rows in this lane's); each
// lane eliminates inside its block downwards and upwards, so that every row i
// reads
//   L_i x_{lo-1} + B_i x_i + R_i x_{hi} = D_i,
// and the 2P-unknown system of the blocks' first and last rows is an affine
// recurrence over the blocks, two divisions in series per block.  On return
// xl, xr are the lane's x_{lo-1} and x_{hi}; the rows follow from them
// elementwise.  NG: negated sub-diagonal, 0 in row 1.
template <class T>
__device__ __forceinline__ T from_f64(double v) { return v; }
template <>
__device__ __forceinline__ float from_f64<float>(double v) { return f64_to_f32_int(v); }

// A quotient of the elimination: FP32 by the branch-free division where it
// holds, FP64 by the ordinary one.
__device__ __forceinline__ float ladder_div(float a, float b) {
    bool ok;
    float q = div_rn(a, b, rcp_rn(b), ok);
    if (!ok) q = div_careful(a, b);
    return q;
}
__device__ __forceinline__ double ladder_div(double a, double b) { return a / b; }
// ok false: the quotient is not valid (ladder_div gives it)
__device__ __forceinline__ float ladder_mid(float a, float b, bool& ok) { return div_mid(a, b, rcp_rn(b), ok); }
__device__ __forceinline__ double ladder_mid(double a, double b, bool& ok) {
    ok = true;
    return a / b;
}

__device__ __forceinline__ void ladder_load2(const float* v, float& a, float& b) {
    const float2 t = *reinterpret_cast<const float2*>(v);
    a = t.x, b = t.y;
}
__device__ __forceinline__ void ladder_load2(const double* v, double& a, double& b) {
    const double2 t = *reinterpret_cast<const double2*>(v);
    a = t.x, b = t.y;
}

// blk: 8 values per block of the recurrence, then 4 results, 16-byte aligned.
template <class T>
__device__ inline void warp_partition_solve(int P, int lane, int len, T* __restrict__ B, T* __restrict__ D,
                                            T* __restrict__ L, T* __restrict__ R, const T* __restrict__ NG,
                                            T* __restrict__ blk, T& xl, T& xr) {
    if (lane < P) {
        // downward: move the sub-diagonal into the left spike L
        T lp = NG[lane], bp = B[lane], dp = D[lane];
        L[lane] = lp;
#pragma unroll 2
        for (int o = 33 + lane, r = 1; r < len; ++r, o += 33) {
            const T a = NG[o];
            bool ok;
            T f = ladder_mid(a, bp, ok);
            if (!ok) f = ladder_div(a, bp);
            lp = -f * lp;
            bp = B[o] - f * a;
            dp = D[o] - f * dp;
            L[o] = lp;
            B[o] = bp;
            D[o] = dp;
        }
        // upward: move the super-diagonal into the right spike R
        T rp = lane + 1 < P ? NG[lane + 1] : (T)0;
        T* v = blk + 8 * lane;  // b0 l0 l1 b1 | -r0 -r1 | d0 d1
        v[2] = lp, v[3] = bp, v[5] = -rp, v[7] = dp;
        R[(len - 1) * 33 + lane] = rp;
        // the diagonal is final here, so four rows' FP32 quotients are taken side by side
        constexpr int kRows = sizeof(T) == 4 ? 4 : 1;
        for (int r = len - 2; r >= 0; r -= kRows) {
            T f[kRows], bn[kRows];
            bool all = true;
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                const int o = (r - u >= 0 ? r - u : 0) * 33 + lane;
                bool ok;
                bn[u] = B[o];
                f[u] = ladder_mid(NG[o + 33], u ? bn[u - 1] : bp, ok);
                all = all && (ok || r - u < 0);
            }
            if (!all) {
#pragma unroll
                for (int u = 0; u < kRows; ++u)
                    if (r - u >= 0) f[u] = ladder_div(NG[(r - u) * 33 + lane + 33], u ? bn[u - 1] : bp);
            }
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if (r - u < 0) break;
                const int o = (r - u) * 33 + lane;
                lp = L[o] - f[u] * lp;
                rp = -f[u] * rp;
                dp = D[o] - f[u] * dp;
                L[o] = lp;
                R[o] = rp;
                D[o] = dp;
                bp = bn[u];
            }
        }
        v[0] = bp, v[1] = lp, v[4] = -rp, v[6] = dp;
    }
    __syncwarp();
    // forward over blocks: l_{j-1} = al + be f_j;  f_j = p_j + q_j f_{j+1};  l_j = al_j + be_j f_{j+1}
    T al = 0, be = 0;
    T* const res = blk + 32 * 8;
    if constexpr (sizeof(T) == 4) {
        // every lane alike; the next block's values are loaded, and its end
        // row's reciprocal taken, while this block's two divisions run
        const float4* v4 = reinterpret_cast<const float4*>(blk);
        float4 u = v4[0], w = v4[1];
        float rb = rcp_rn(u.w);
        for (int j = 0; j < P; ++j) {
            const int jn = j + 1 < P ? j + 1 : j;
            const float4 un = v4[2 * jn], wn = v4[2 * jn + 1];
            const float rbn = rcp_rn(un.w);
            const float den = u.x + u.y * be, rd = rcp_rn(den), lb = u.z * be;
            const float pn = w.z - u.y * al, an = w.w - u.z * al;
            bool ok0, ok1, ok2, ok3;
            float q = div_rn(w.x, den, rd, ok0), p = div_rn(pn, den, rd, ok1);
            float nb = div_rn(w.y - lb * q, u.w, rb, ok2), na = div_rn(an - lb * p, u.w, rb, ok3);
            if (!(ok0 && ok1 && ok2 && ok3)) {  // the same in every lane
                q = div_careful(w.x, den), p = div_careful(pn, den);
                nb = div_careful(w.y - lb * q, u.w), na = div_careful(an - lb * p, u.w);
            }
            if (lane == 0) reinterpret_cast<float4*>(res)[j] = make_float4(q, nb, p, na);
            al = na;
            be = nb;
            u = un, w = wn, rb = rbn;
        }
    } else {
        // even lanes carry q and be, odd lanes p and al: the same two divisions
        const int odd = lane & 1;
        for (int j = 0; j < P; ++j) {
            const T* v = blk + 8 * j;
            T b0, l0, l1, b1, x0, x1;
            ladder_load2(v, b0, l0), ladder_load2(v + 2, l1, b1), ladder_load2(v + 4 + 2 * odd, x0, x1);
            const T den = b0 + l0 * be, lb = l1 * be;
            const T q = (odd ? x0 - l0 * al : x0) / den;
            const T n = ((odd ? x1 - l1 * al : x1) - lb * q) / b1;
            if (lane < 2) res[4 * j + 2 * odd] = q, res[4 * j + 2 * odd + 1] = n;  // q nb p na
            al = n;
            be = __shfl_sync(0xffffffffu, n, 0);
        }
    }
    __syncwarp();
    // backward: f_P = 0
    T fnext = 0, last = 0;
    xr = 0;
#pragma unroll 4
    for (int j = P - 1; j >= 0; --j) {
        const T* v = res + 4 * j;
        T qj, nb, pj, na;
        ladder_load2(v, qj, nb), ladder_load2(v + 2, pj, na);
        if (lane == j) xr = fnext, last = na + nb * fnext;
        fnext = pj + qj * fnext;
    }
    xl = __shfl_up_sync(0xffffffffu, last, 1);
    if (lane == 0) xl = 0;
}

// Scalars of one step, thread 0's for the CTA.
struct LadderCtl {
    double V, h, r_hg, hg, a1, a2, b0h2, r_b0h2, r_h, r_2h;
    int go;
    unsigned idx;
};
static_assert(sizeof(LadderCtl) <= 16 * 8, "the control block fits its slot");

template <int PREC, bool WS>
__global__ void __launch_bounds__(128, 4) ladder_kernel(LadderLaunch L) {
    using T = typename std::conditional<PREC == SP_PREC_MIXED, float, double>::type;
    constexpr bool kExact = PREC == SP_PREC_FP64_EXACT, mx = PREC == SP_PREC_MIXED;
    extern __shared__ __align__(16) unsigned char lsm[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nt = blockDim.x;
    const sp_ladder_config& c = L.cfg;
    const int S = c.max_sections + 2, SL = ladder_solve_len(c.max_sections, PREC);
    double* dsm = reinterpret_cast<double*>(lsm);
    LadderCtl& ctl = *reinterpret_cast<LadderCtl*>(dsm);
    unsigned long long* red = reinterpret_cast<unsigned long long*>(dsm + 16);  // [2][8]
    T* blk = reinterpret_cast<T*>(dsm + kLadderCtl);
    double* A0 = reinterpret_cast<double*>(blk + kLadderBlk);
    double* A = WS ? L.ws + (size_t)blockIdx.x * LA_COUNT * S : A0;
    double *g = A + LA_G * S, *C = A + LA_C * S, *x = A + LA_X * S, *ip = A + LA_IP * S, *xs = A + LA_XS * S;
    double *geq = A + LA_GEQ * S, *ieq = A + LA_IEQ * S;
    T* ts = reinterpret_cast<T*>(A0 + (WS ? 0 : LA_COUNT * S));
    T *sB = ts + LS_B * SL, *sD = ts + LS_D * SL, *sL = ts + LS_L * SL, *sR = ts + LS_R * SL, *sNG = ts + LS_NG * SL;
    T *sJ = ts + LS_J * SL, *fl = ts + LS_COUNT * SL;  // fl: [32] x_{lo-1}, [32] x_{hi}
    uint32_t* at = reinterpret_cast<uint32_t*>(lsm + (((unsigned char*)(fl + 64) - lsm + 7) & ~(ptrdiff_t)7));
    unsigned hard = 0;
    const double nvt = c.diode_n * thermal_voltage_300();
    const double inv_nvt = 1.0 / nvt;
    const double vcrit = nvt * cr_log(nvt / (1.4142135623730951 * 1e-14), &hard);
    const double gamma = 2.0 - 1.4142135623730951;
    const float inv_nvt_f = f64_to_f32_int(inv_nvt), is_f = f64_to_f32_int(c.diode_is);
    const float vrel = f64_to_f32_int(c.v_reltol), vabs = f64_to_f32_int(c.v_abstol);
    const double inv_per = 1.0 / c.pulse.per;
    const int ldx = c.max_sections + 2;

    // vd > vcrit for vcrit > 0 from the bit patterns (a NaN counts as above: its
    // limited value is NaN too), so that the test does not take the FP64 pipe
    const long long kcrit = vcrit > 0.0 ? __double_as_longlong(vcrit) : -1;
    auto above = [&](double vd) { return kcrit >= 0 ? __double_as_longlong(vd) > kcrit : vd > vcrit; };
    auto limit = [&](double vd) {
        if (above(vd)) {
            if (kExact) {
                const double arg = (vd - vcrit) / nvt;
                return vcrit + nvt * (1.0 + pm_log1p(arg, &hard));
            }
            return vcrit + nvt * (1.0 + log1p((vd - vcrit) * inv_nvt));
        }
        return vd;
    };
    // exp of the diode: the portable correctly rounded one for the exact mode,
    // the device's (shorter dependency chain) otherwise
    auto dexp = [&](double v) { return kExact ? cr_exp(v / nvt, &hard) : exp(v * inv_nvt); };
    // largest of the CTA's non-negative values (order-preserving bit patterns)
    auto warp_max = [&](double v) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(v);
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32));
        const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(b >> 32) == hi ? (unsigned)b : 0u);
        return ((unsigned long long)hi << 32) | lo;
    };

    while (true) {
        if (tid == 0) ctl.idx = atomicAdd(L.next, 1u);
        __syncthreads();
        const unsigned idx = ctl.idx;
        if (idx >= L.count) break;
        const uint32_t i = L.order[idx];
        const uint32_t inst = (uint32_t)(L.first + i);
        const int N = ladder_sections(c, L.seed, inst);
        const int P = N / 2 < 32 ? N / 2 : 32;
        int len = 0;  // rows of this lane's block
        // draws (a exp(u ln(b/a)), the log-uniform rule of the parameter draws) and the DC start (all zero)
        const double lr = cr_log(c.r_hi / c.r_lo, &hard), lc = cr_log(c.c_hi / c.c_lo, &hard);
        for (int k = 1 + tid; k <= N; k += nt) {
            const double Rk = c.r_lo * cr_exp(rng_uniform(L.seed, inst, 2u * k - 1u) * lr, &hard);
            C[k] = c.c_lo * cr_exp(rng_uniform(L.seed, inst, 2u * k) * lc, &hard);
            g[k] = 1.0 / Rk;
            ip[k] = 0.0;
            x[k] = 0.0;
            if (kExact) at[k] = (uint32_t)k;
        }
        if (tid == 0) x[0] = x[N + 1] = 0.0;
        if (lane < P) {  // block b: rows 1 + b N / P .. ; every warp places a share of its rows
            const unsigned lo = 1u + (unsigned)lane * (unsigned)N / (unsigned)P;
            const unsigned hi = 1u + (unsigned)(lane + 1) * (unsigned)N / (unsigned)P;
            len = (int)(hi - lo);
            if (!kExact)
                for (int r = wid; r < len; r += nt >> 5)
                    at[lo + r] = ((uint32_t)lane << 16) | (uint32_t)(r * 33 + lane);
        }
        __syncthreads();
        if (!kExact)
            for (int k = 1 + tid; k <= N; k += nt) sNG[at[k] & 0xffffu] = k > 1 ? -from_f64<T>(g[k]) : (T)0;
        // thread 0's: time, step, counters
        double t = 0.0, h = c.h_init;
        int accepted = 0, rejected = 0, iterations = 0, steps = 0, next_probe = 0;
        uint8_t status = SP_ST_CONVERGED;
        double* probe = L.probe ? L.probe + (size_t)i * c.num_probe : nullptr;
        double tp = 0.0;  // time of probe next_probe
        auto record = [&](double t0, double xa, double t1, double xb) {
            while (next_probe < c.num_probe && !(tp > t1)) {
                if (probe) probe[next_probe] = t1 > t0 ? xa + (xb - xa) * ((tp - t0) / (t1 - t0)) : xb;
                ++next_probe;
                tp = c.num_probe > 1 ? c.tstop * (double)next_probe / (double)(c.num_probe - 1) : 0.0;
            }
        };
        // the stage's companions: conductance ge(k), then the constant part of the diagonal
        auto companions = [&](auto ge, auto ie) {
            for (int k = 1 + tid; k <= N; k += nt) {
                const double gq = ge(k);
                geq[k] = gq;
                ieq[k] = ie(k, gq);
                const double gk1 = k < N ? g[k + 1] : 0.0;
                sJ[at[k] & 0xffffu] = from_f64<T>((g[k] + gk1) + gq);
            }
        };
        // Newton solve of a stage from xs: iterations (> 0), -1 on a miss, -2 on NaN/Inf
        auto newton = [&](double V) -> int {
            for (int it = 1; it <= c.max_iterations; ++it) {
                for (int k = 1 + tid; k <= N; k += nt) {
                    const int w = (int)(at[k] & 0xffffu);
                    if (!mx) {
                        // full-step form: diag and rhs of the linearised stage (oracle order)
                        const double vl1 = limit(xs[k]);
                        const double vl2 = limit(vl1);
                        const double e = dexp(vl2);
                        const double id = c.diode_is * (e - 1.0);
                        const double gd = kExact ? fmax(c.diode_is * e / nvt, 1e-12) : fmax(c.diode_is * e * inv_nvt, 1e-12);
                        const double ieq_d = id - gd * vl1;
                        sB[w] = (T)(sJ[w] + gd);
                        double r = (0.0 + ieq[k]) - ieq_d;
                        if (k == 1) r = r - (-g[1]) * V;
                        sD[w] = (T)r;
                    } else {
                        // correction form: FP64 residual of the linearised stage, FP32 solve.
                        // exp(a) = expf(ah) (1 + al), a = ah + al split at FP32 (relative error
                        // ~1e-7, far inside the stage tolerances), conductance and Jacobian in
                        // FP32, conversions on the integer pipe: the FP64 pipe keeps only the
                        // residual (what the refinement needs) and the update
                        const double xk = xs[k];
                        const bool lim = above(xk);
                        const double vl1 = limit(xk);
                        const double vl2 = lim ? limit(vl1) : vl1;
                        const double a = vl2 * inv_nvt;
                        const float ah = f64_to_f32_int(a);
                        const float ef = expf(ah);
                        const double e = f32_to_f64_int(ef) * (1.0 + (a - f32_to_f64_int(ah)));
                        double id = c.diode_is * (e - 1.0);
                        const float gdf = fmaxf(is_f * ef * inv_nvt_f, 1e-12f);
                        const double xlk = k == 1 ? V : xs[k - 1];
                        const double xrk = k < N ? xs[k + 1] : 0.0;
                        const double gk1 = k < N ? g[k + 1] : 0.0;
                        // KCL: currents leaving node k (R left, R right, C companion, diode linearised at vl1)
                        if (lim) id = id + f32_to_f64_int(gdf) * (xk - vl1);  // xk - vl1 is 0 otherwise
                        const double F = g[k] * (xk - xlk) + gk1 * (xk - xrk) + (geq[k] * xk - ieq[k]) + id;
                        sB[w] = sJ[w] + gdf;
                        sD[w] = __uint_as_float(__float_as_uint(f64_to_f32_int(F)) ^ 0x80000000u);
                    }
                }
                __syncthreads();
                if (kExact) {
                    if (tid == 0) {
                        sL[1] = (N > 1 ? -g[2] : 0.0) / sB[1];
                        sR[1] = sD[1] / sB[1];
                        for (int k = 2; k <= N; ++k) {
                            const double sub = -g[k];
                            const double m = sB[k] - sub * sL[k - 1];
                            sL[k] = (k < N ? -g[k + 1] : 0.0) / m;
                            sR[k] = (sD[k] - sub * sR[k - 1]) / m;
                        }
                        // back substitution into sD (the new iterate of nodes 1..N)
                        sD[N] = sR[N];
                        for (int k = N - 1; k >= 1; --k) sD[k] = sR[k] - sL[k] * sD[k + 1];
                    }
                } else if (wid == 0) {
                    T xl, xr;
                    warp_partition_solve<T>(P, lane, len, sB, sD, sL, sR, sNG, blk, xl, xr);
                    fl[lane] = xl;
                    fl[32 + lane] = xr;
                }
                __syncthreads();
                bool ok = true, fin = true;
                for (int k = 1 + tid; k <= N; k += nt) {
                    const uint32_t bw = at[k];
                    const int w = (int)(bw & 0xffffu), b = (int)(bw >> 16);
                    T dn = sD[w];
                    if (!kExact) {
                        dn = ladder_div(sD[w] - sL[w] * fl[b] - sR[w] * fl[32 + b], sB[w]);
                    }
                    const double old = xs[k];
                    if (!mx) {
                        const double nw = dn;
                        const double tol = c.v_reltol * fmax(fabs(nw), fabs(old)) + c.v_abstol;
                        ok = ok && fabs(nw - old) <= tol;
                        fin = fin && isfinite(nw);
                        xs[k] = nw;
                    } else {
                        const float dy = (float)dn;
                        const double nw = old + f32_to_f64_int(dy);
                        const float nwf = f64_to_f32_int(nw), oldf = f64_to_f32_int(old);
                        ok = ok && !(fabsf(dy) > vrel * fmaxf(fabsf(nwf), fabsf(oldf)) + vabs);
                        fin = fin && isfinite(nwf);
                        xs[k] = nw;
                    }
                }
                if (tid == 0) {
                    // source node and branch current (KCL of node in)
                    const double v0 = xs[0], i0 = xs[N + 1];
                    const double inew = -(g[1] * V + (-g[1]) * xs[1]);
                    if (__double_as_longlong(V) != __double_as_longlong(v0))  // the first iteration only
                        ok = ok && fabs(V - v0) <= c.v_reltol * fmax(fabs(V), fabs(v0)) + c.v_abstol;
                    ok = ok && fabs(inew - i0) <= c.v_reltol * fmax(fabs(inew), fabs(i0)) + c.i_abstol;
                    fin = fin && isfinite(inew);
                    xs[0] = V;
                    xs[N + 1] = inew;
                }
                if (__syncthreads_and(ok && fin)) return it;
                if (!__syncthreads_and(fin)) return -2;
            }
            return -1;
        };
        if (tid == 0) record(0.0, 0.0, 0.0, 0.0);
        while (true) {
            if (wid == 0) {
                // the scalars of the step: warp 0's lanes hold thread 0's h and divide
                // side by side (an FP64 instruction takes a warp 64 cycles, so divisions
                // in one thread would be in series)
                int go = 0;
                if (lane == 0 && t < c.tstop) {
                    if (++steps > c.max_steps) {
                        status = SP_ST_FAILED;
                    } else {
                        go = 1;
                        h = fmin(fmax(h, c.h_min), c.h_max);
                        if (t + h > c.tstop) h = c.tstop - t;
                    }
                }
                go = __shfl_sync(0xffffffffu, go, 0);
                if (go) {
                    const double hb = __shfl_sync(0xffffffffu, h, 0);
                    const double hg = gamma * hb, h2 = (1.0 - gamma) * hb, h1 = gamma * hb;
                    // MIXED: one reciprocal per step instead of a divide per node (GB300's
                    // FP64 divide is a long FP64-pipe sequence); the other modes keep the
                    // reference's 2 C / (gamma h) per node
                    const double q1 = (lane == 0 ? 2.0 : lane == 1 ? h2 : lane == 2 ? 1.0 : 2.0) /
                                      (lane == 0 ? hg : lane == 1 ? h1 : hb);
                    const double rho = __shfl_sync(0xffffffffu, q1, 1);
                    const double denom = 1.0 + 2.0 * rho;
                    const double q2 = (lane == 0 ? (1.0 + rho) * (1.0 + rho) : lane == 1 ? -rho * rho : 1.0 + rho) / denom;
                    const double b0h2 = __shfl_sync(0xffffffffu, q2, 2) * h2;
                    if (lane == 0) {
                        ctl.h = hb, ctl.hg = hg, ctl.r_hg = q1, ctl.a1 = q2;
                        ctl.V = ladder_pulse(c.pulse, t + hb, inv_per);
                        ctl.b0h2 = b0h2;
                        ctl.r_b0h2 = 1.0 / b0h2;
                    }
                    if (lane == 1) ctl.a2 = q2;
                    if (lane == 2) ctl.r_h = q1;
                    if (lane == 3) ctl.r_2h = q1;
                }
                if (lane == 0) ctl.go = go;
            }
            __syncthreads();
            if (!ctl.go) break;
            const double V = ctl.V, hs = ctl.h;
            {
                const double hg = ctl.hg, r_hg = ctl.r_hg;
                companions([&](int k) { return mx ? C[k] * r_hg : 2.0 * C[k] / hg; },
                           [&](int k, double gq) { return gq * x[k] + ip[k]; });
            }
            for (int k = tid; k <= N + 1; k += nt) xs[k] = x[k];
            __syncthreads();
            const int it1 = newton(V);
            int it2 = -1;
            if (it1 > 0) {
                const double a1 = ctl.a1, a2 = ctl.a2, b0h2 = ctl.b0h2, r_b0h2 = ctl.r_b0h2;
                // the intermediate stage's solution is xs, the step's start x
                companions([&](int k) { return mx ? C[k] * r_b0h2 : C[k] / b0h2; },
                           [&](int k, double gq) { return gq * (a1 * xs[k] + a2 * x[k]); });
                it2 = newton(V);
            }
            if (it1 == -2 || it2 == -2) {
                if (tid == 0) {
                    status = SP_ST_NONFINITE;
                    if (it1 > 0) iterations += it1;
                }
                break;
            }
            if (it1 < 0 || it2 < 0) {
                if (tid == 0) {
                    if (it1 > 0) iterations += it1;
                    ++rejected;
                    if (h <= c.h_min) status = SP_ST_FAILED;
                    else h *= 0.25;
                }
                if (hs <= c.h_min) break;
                continue;
            }
            double lte = 0.0, ref = 0.0;
            const double r_h = ctl.r_h, r_2h = ctl.r_2h;
            for (int k = 1 + tid; k <= N; k += nt) {
                const double v_new = xs[k];
                const double i_trap = (mx ? C[k] * r_2h : 2.0 * C[k] / hs) * (v_new - x[k]) - ip[k];
                const double i_be = (mx ? C[k] * r_h : C[k] / hs) * (v_new - x[k]);
                lte = fmax(lte, mx ? fabs(i_trap - i_be) * (1.0 / 3.0) : fabs(i_trap - i_be) / 3.0);
                ref = fmax(ref, fabs(v_new));
            }
            {
                const unsigned long long wl = warp_max(lte), wr = warp_max(ref);
                if (lane == 0) red[wid] = wl, red[8 + wid] = wr;
            }
            __syncthreads();
            unsigned long long ml = 0, mr = 0;
            for (int q = 0; q < nt >> 5; ++q) {
                ml = red[q] > ml ? red[q] : ml;
                mr = red[8 + q] > mr ? red[8 + q] : mr;
            }
            const double max_lte = __longlong_as_double((long long)ml), max_ref = __longlong_as_double((long long)mr);
            const double tol = fmax(c.lte_abstol, c.lte_reltol * max_ref);
            if (max_lte > tol && hs > c.h_min) {
                if (tid == 0) {
                    iterations += it1 + it2;
                    ++rejected;
                    h *= fmax(fmin(sqrt(tol / max_lte), 0.5), 0.1);
                }
                continue;
            }
            const double xa = x[N], xb = xs[N];
            __syncthreads();  // thread 0 has read x[N]
            if (tid == 0) {
                record(t, xa, t + h, xb);
                iterations += it1 + it2;
                if (L.steps && accepted < L.max_rec) L.steps[(size_t)i * L.max_rec + accepted] = h;
                t += h;
                ++accepted;
                if (max_lte < tol * 0.5 && h < c.h_max) h *= fmin(fmin(sqrt(tol / fmax(max_lte, 1e-20)), 2.0), 1.5);
            }
            for (int k = 1 + tid; k <= N; k += nt) {
                ip[k] = geq[k] * xs[k] - ieq[k];
                x[k] = xs[k];
            }
            if (tid == 0) {
                x[0] = xs[0];
                x[N + 1] = xs[N + 1];
            }
        }
        __syncthreads();
        double* xf = L.x_final + (size_t)i * ldx;
        for (int k = tid; k < ldx; k += nt) xf[k] = k <= N + 1 ? x[k] : 0.0;
        if (tid == 0) {
            while (next_probe < c.num_probe) {
                if (probe) probe[next_probe] = x[N];
                ++next_probe;
            }
            L.n[i] = N + 2;
            L.accepted[i] = accepted;
            L.rejected[i] = rejected;
            L.iters[i] = iterations;
            L.status[i] = status;
        }
        __syncthreads();
    }
}

}  // namespace SP_KERNEL_NS
#endif  // SP_KERNEL_NS

}  // namespace sp
