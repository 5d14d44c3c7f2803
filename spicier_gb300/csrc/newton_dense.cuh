// Batched dense Newton-Raphson DC operating points, one thread per sample.
//
// Follows solve_newton_raphson (crates/spicier-solver/src/newton.rs:70-131):
// restamp at the current iterate, solve the linearised system, test the step
// with check_convergence (newton.rs:134-159), take the full step; gmin and
// source stepping (newton.rs:261-459) are the fallback chain.
//
// Work layout: every per-sample array lives in shared memory, interleaved
// across the threads of the block (element i of thread t at
// base[i * blockDim + t]), so each warp-wide access touches 32 consecutive
// words: no bank conflicts for FP32 and two wavefronts for FP64.
//
// Precision modes (template PREC):
//   SP_PREC_FP64  — the reference's arithmetic: the FP64 system A x_new = b
//                   is factorised with the same partial-pivot LU as
//                   nalgebra's LU::new/solve (column icamax pivot, multipliers
//                   scaled by 1/diag, column-oriented axpy updates).  Built
//                   without FMA contraction it is bit-identical to the
//                   reference on circuits without transcendental models.
//   SP_PREC_MIXED — correction form: the FP64 KCL residual F(x) = A(x)x - b(x)
//                   is accumulated from the stamps, the Jacobian A(x) is
//                   stored and factorised in FP32, delta = -A32^-1 F is taken
//                   in FP32 and the update x += delta, the convergence test
//                   and the device models stay FP64.  Newton itself is the
//                   FP64 iterative refinement: the fixed point is the FP64
//                   root of F, independent of the FP32 factorisation error.
#pragma once
#include "circuit_dev.cuh"
#include "draw.cuh"
#include "pdl.cuh"

namespace sp {

// a / b as IEEE division gives it, on the integer pipe wherever both operands
// and the quotient are normal (a quotient of a zero is that zero with the
// operands' sign), in hardware otherwise.
__device__ __forceinline__ double div_int(double a, double b) {
    const uint64_t sign = (cr::dbits(a) ^ cr::dbits(b)) & (1ULL << 63);
    const double q = ieee_div(fabs(a), fabs(b));
    return cr::bdouble((cr::dbits(q) & ~(1ULL << 63)) | sign);
}

template <class T>
struct Il {  // interleaved per-thread array view
    T* base;
    int bs;
    __device__ T& operator[](int i) const { return base[(size_t)i * bs]; }
};

struct PlainSink {
    static constexpr bool kTeam = false;
    Il<double> A, b, xs;
    int n;
    __device__ double x(int i) const { return xs[i]; }
    __device__ void add(int r, int c, double v) { A[c * n + r] += v; }
    __device__ void rhs_add(int r, double v) { b[r] += v; }
    __device__ void rhs_set(int r, double v) { b[r] = v; }
};

// Jacobian in FP32, residual F = A x - b in FP64 (only one element writes a
// branch row's RHS, so rhs_set is a subtraction from zero).
struct MixedSink {
    static constexpr bool kTeam = false;
    Il<float> J;
    Il<double> F, xs;
    int n;
    __device__ double x(int i) const { return xs[i]; }
    __device__ void add(int r, int c, double v) {
        J[c * n + r] += (float)v;
        F[r] += v * xs[c];
    }
    __device__ void rhs_add(int r, double v) { F[r] -= v; }
    __device__ void rhs_set(int r, double v) { F[r] -= v; }
};

struct ResidSink {
    static constexpr bool kTeam = false;
    Il<double> F, xs;
    __device__ double x(int i) const { return xs[i]; }
    __device__ void add(int r, int c, double v) { F[r] += v * xs[c]; }
    __device__ void rhs_add(int r, double v) { F[r] -= v; }
    __device__ void rhs_set(int r, double v) { F[r] -= v; }
};

// PlainSink and MixedSink that also record which entries of the matrix the
// circuit stamps: lane c of the warp holds the rows of column c in `rows`
// (every lane of the warp stamps the same circuit).
struct PlainSinkRec : PlainSink {
    static constexpr bool kIntTests = true;
    int lane;
    unsigned rows = 0;
    __device__ PlainSinkRec(Il<double> A_, Il<double> b_, Il<double> x_, int n_, int l) : PlainSink{A_, b_, x_, n_}, lane(l) {}
    __device__ void mark(int r, int c) {
        if (c == lane) rows |= 1u << r;
    }
    __device__ void add(int r, int c, double v) {
        PlainSink::add(r, c, v);
        mark(r, c);
    }
};
struct MixedSinkRec : MixedSink {
    static constexpr bool kIntTests = true;
    int lane;
    unsigned rows = 0;
    __device__ MixedSinkRec(Il<float> J_, Il<double> F_, Il<double> x_, int n_, int l) : MixedSink{J_, F_, x_, n_}, lane(l) {}
    __device__ void add(int r, int c, double v) {
        MixedSink::add(r, c, v);
        if (c == lane) rows |= 1u << r;
    }
};

// A sink, or (TEAM) the same for a sample that `team` lanes hold; lanes: those
// that stamp together, one team where teams go their own ways or the whole warp.
template <class S>
struct TeamSink : S {
    static constexpr bool kTeam = true;
    int team;
    unsigned lanes;
    template <class... A>
    __device__ TeamSink(int t, unsigned l, A... a) : S{a...}, team(t), lanes(l) {}
};
template <bool TEAM, class S, class... A>
__device__ inline auto make_sink(int team, unsigned lanes, A... a) {
    if constexpr (TEAM) return TeamSink<S>(team, lanes, a...);
    else return S{a...};
}

// MOSFET stamps with their eight loads in flight together (one after the
// other, each waits for the store before it) where no two entries coincide;
// each entry takes the additions of stamp_mos in its order.
__device__ inline void stamp_mos(PlainSinkRec& k, int d, int g, int so, double gds, double gm, double ieq) {
    if (d < 0 || g < 0 || so < 0 || d == g || d == so || g == so) {
        stamp_mos<PlainSinkRec>(k, d, g, so, gds, gm, ieq);
        return;
    }
    const int n = k.n;
    double &add = k.A[d * n + d], &ass = k.A[so * n + so], &ads = k.A[so * n + d], &asd = k.A[d * n + so];
    double &adg = k.A[g * n + d], &asg = k.A[g * n + so], &bd = k.b[d], &bs = k.b[so];
    const double v0 = add, v1 = ass, v2 = ads, v3 = asd, v4 = adg, v5 = asg, v6 = bd, v7 = bs;
    add = v0 + gds;
    ass = (v1 + gds) + gm;
    ads = (v2 - gds) - gm;
    asd = v3 - gds;
    adg = v4 + gm;
    asg = v5 - gm;
    bd = v6 - ieq;
    bs = v7 + ieq;
    k.mark(d, d), k.mark(so, so), k.mark(d, so), k.mark(so, d), k.mark(d, g), k.mark(so, g);
}

// nalgebra-order partial-pivot LU of A in place (column-major, A[c*n+r]); the
// row permutation is applied to b as it is found, which is the order in which
// LU::solve replays it.  A zero on the diagonal afterwards: singular.
__device__ inline void lu_factor_fp64(int n, Il<double> A, Il<double> b) {
    for (int i = 0; i < n; ++i) {
        int piv = i;
        double best = fabs(A[i * n + i]);
        for (int r = i + 1; r < n; ++r) {
            double v = fabs(A[i * n + r]);
            if (v > best) {
                best = v;
                piv = r;
            }
        }
        double diag = A[i * n + piv];
        if (diag == 0.0) continue;
        if (piv != i) {
            for (int c = 0; c < n; ++c) {
                double t = A[c * n + i];
                A[c * n + i] = A[c * n + piv];
                A[c * n + piv] = t;
            }
            double t = b[i];
            b[i] = b[piv];
            b[piv] = t;
        }
        double inv = 1.0 / diag;
        for (int r = i + 1; r < n; ++r) A[i * n + r] = A[i * n + r] * inv;
        for (int c = i + 1; c < n; ++c) {
            double p = A[c * n + i];
            for (int r = i + 1; r < n; ++r) A[c * n + r] = -p * A[i * n + r] + A[c * n + r];
        }
    }
}

// The solve: factorisation, then b overwritten by x.  Returns false on a zero
// pivot (the system is singular).
__device__ inline bool lu_solve_fp64(int n, Il<double> A, Il<double> b) {
    lu_factor_fp64(n, A, b);
    for (int i = 0; i < n; ++i) {
        double coeff = b[i];
        for (int r = i + 1; r < n; ++r) b[r] = -coeff * A[i * n + r] + b[r];
    }
    for (int i = n - 1; i >= 0; --i) {
        double diag = A[i * n + i];
        if (diag == 0.0) return false;
        double coeff = b[i] / diag;
        b[i] = coeff;
        for (int r = 0; r < i; ++r) b[r] = -coeff * A[i * n + r] + b[r];
    }
    return true;
}

// FP32 partial-pivot LU solve (same algorithm, FMA allowed).
__device__ inline bool lu_solve_fp32(int n, Il<float> A, Il<float> b) {
    for (int i = 0; i < n; ++i) {
        int piv = i;
        float best = fabsf(A[i * n + i]);
        for (int r = i + 1; r < n; ++r) {
            float v = fabsf(A[i * n + r]);
            if (v > best) {
                best = v;
                piv = r;
            }
        }
        float diag = A[i * n + piv];
        if (diag == 0.0f) continue;
        if (piv != i) {
            for (int c = 0; c < n; ++c) {
                float t = A[c * n + i];
                A[c * n + i] = A[c * n + piv];
                A[c * n + piv] = t;
            }
            float t = b[i];
            b[i] = b[piv];
            b[piv] = t;
        }
        float inv = 1.0f / diag;
        for (int r = i + 1; r < n; ++r) A[i * n + r] *= inv;
        for (int c = i + 1; c < n; ++c) {
            float p = A[c * n + i];
            for (int r = i + 1; r < n; ++r) A[c * n + r] = fmaf(-p, A[i * n + r], A[c * n + r]);
        }
    }
    for (int i = 0; i < n; ++i) {
        float coeff = b[i];
        for (int r = i + 1; r < n; ++r) b[r] = fmaf(-coeff, A[i * n + r], b[r]);
    }
    for (int i = n - 1; i >= 0; --i) {
        float diag = A[i * n + i];
        if (diag == 0.0f) return false;
        float coeff = b[i] / diag;
        b[i] = coeff;
        for (int r = 0; r < i; ++r) b[r] = fmaf(-coeff, A[i * n + r], b[r]);
    }
    return true;
}

// 2^-500 <= |x| < 2^500
__device__ __forceinline__ bool mid_range(double x) {
    return (((unsigned)(__double_as_longlong(x) >> 32) & 0x7fffffffu) >> 20) - 523u < 1000u;
}

// a / b as IEEE division gives it, given r = 1 / b: two correction steps of the
// fused remainder (Markstein: r correctly rounded makes the second one round
// a / b correctly), five FP64 instructions instead of a division's ten, where
// every step stays normal; the division elsewhere.
__device__ __forceinline__ double warp_div(double a, double b, double r) {
    const double q0 = a * r;
    double q = fma(fma(-b, q0, a), r, q0);
    q = fma(fma(-b, q, a), r, q);
    if (!(mid_range(a) && mid_range(b))) q = __double_as_longlong(a) << 1 == 0 && mid_range(b) ? q0 : a / b;
    return q;
}
__device__ __forceinline__ float warp_div(float a, float b, float) { return a / b; }
__device__ __forceinline__ bool finite_bits(double x) { return ((unsigned)(__double_as_longlong(x) >> 32) & 0x7ff00000u) != 0x7ff00000u; }
__device__ __forceinline__ bool finite_bits(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ unsigned long long abs_bits(double x) { return (unsigned long long)__double_as_longlong(x) & ~(1ULL << 63); }
__device__ __forceinline__ unsigned abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// lu_solve_fp64 / lu_solve_fp32 of the 32 samples of a warp (n <= 32), leaving
// out the entries that are zero in all of them.  rows: lane c's mask of the
// rows of column c that may be nonzero.  The mask follows the row swaps (a
// union of the lanes' choices where they differ) and the fill, every loop runs
// over set bits alike in all lanes, and every entry takes the operations of
// the dense solve in the same order but for additions of a zero product; the
// right-hand side is eliminated along (its multipliers need no storage).
// False: the lane's system is singular.  *plain is cleared where a value is
// not finite (a skipped product with a zero would be a NaN): the caller then
// repeats that sample with the dense solve.
//
// Bound: the FP64 pipe (64 cycles per warp instruction), so nothing else runs
// on it: the pivot search compares bit patterns, the substitution's quotients
// come from the pivots' reciprocals, and pivots of +-1 (voltage-source rows)
// divide nothing.  The op-amp's 12 x 12 matrix takes about 100 of the dense
// 780 updates; its 65,536-sample FP64 sweep went from 1,447 to 583 us, the
// 1,024-sample 5-unknown amplifier's from 85 to 66.
template <class T>
__device__ inline bool lu_solve_warp(int n, int lane, Il<T> A, Il<T> b, unsigned rows, bool* plain) {
    bool ok = true, fin = true;
    unsigned ones = 0;  // pivots that are +-1 in every lane
    T inv_last = (T)0;
    for (int i = 0; i < n; ++i) {
        const unsigned below = ~((2u << i) - 1u);
        unsigned m = __shfl_sync(0xffffffffu, rows, i) & below;
        auto best = abs_bits(A[i * n + i]);
        int piv = i;
        for (unsigned q = m; q; q &= q - 1) {
            const int r = __ffs(q) - 1;
            const auto v = abs_bits(A[i * n + r]);
            if (v > best) best = v, piv = r;
        }
        // row swap in the columns from i on and in b
        const unsigned pset = __reduce_or_sync(0xffffffffu, 1u << piv);
        const unsigned both = pset | (1u << i);
        if (pset != 1u << i) {
            for (unsigned q = __ballot_sync(0xffffffffu, (rows & both) != 0) & ~((1u << i) - 1u); q; q &= q - 1) {
                const int c = __ffs(q) - 1;
                const T u = A[c * n + i], v = A[c * n + piv];
                A[c * n + i] = v;
                A[c * n + piv] = u;
            }
            const T u = b[i], v = b[piv];
            b[i] = v;
            b[piv] = u;
            if (__popc(pset) == 1) {  // one choice: the two rows' bits change places
                const unsigned p = __ffs(pset) - 1, d = ((rows >> i) ^ (rows >> p)) & 1u;
                rows ^= (d << i) | (d << p);
            } else if (rows & both) {
                rows |= both;
            }
            m = __shfl_sync(0xffffffffu, rows, i) & below;
        }
        const T diag = A[i * n + i];
        T inv = diag;
        if (__all_sync(0xffffffffu, diag == (T)1 || diag == (T)-1)) {
            ones |= 1u << i;
        } else {
            ok = ok && best != 0;
            inv = best != 0 ? (T)1 / diag : (T)0;
        }
        const unsigned cols = __ballot_sync(0xffffffffu, (rows >> i) & 1u) & below;
        const T bi = b[i];
        // four rows of the trailing block at a time, so that their updates overlap
        for (unsigned q = m; q;) {
            int r[4];
            T l[4], br[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                r[u] = q ? __ffs(q) - 1 : -1;
                q &= q - 1;
                const int ru = r[u] < 0 ? i : r[u];
                l[u] = A[i * n + ru];
                br[u] = b[ru];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (r[u] < 0) continue;
                l[u] = l[u] * inv;
                b[r[u]] = -bi * l[u] + br[u];
            }
            for (unsigned cq = cols; cq; cq &= cq - 1) {
                const int c = __ffs(cq) - 1;
                const T p = A[c * n + i];
                T a[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u] = A[c * n + (r[u] < 0 ? i : r[u])];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (r[u] >= 0) A[c * n + r[u]] = -p * l[u] + a[u];
            }
        }
        if ((cols >> lane) & 1u) rows |= m;
        // kept for the back substitution where column i's multipliers were
        if (i + 1 < n) A[i * n + i + 1] = inv;
        else inv_last = inv;
    }
    for (int i = n - 1; i >= 0; --i) {
        T acc = b[i];
        for (unsigned q = __ballot_sync(0xffffffffu, (rows >> i) & 1u) & ~((2u << i) - 1u); q;) {
            const int c = 31 - __clz(q);
            q ^= 1u << c;
            acc = -b[c] * A[c * n + i] + acc;
        }
        const T diag = A[i * n + i];
        const T inv = i + 1 < n ? A[i * n + i + 1] : inv_last;
        acc = (ones >> i) & 1u ? acc * diag : (diag == (T)0 ? (T)0 : warp_div(acc, diag, inv));
        fin = fin && finite_bits(acc);
        b[i] = acc;
    }
    *plain = *plain && fin;
    return ok;
}

// The lanes that hold a sample together with this one (a power of two of them).
__device__ __forceinline__ unsigned team_lanes(unsigned team) {
    return (team == 32 ? 0xffffffffu : (1u << team) - 1u) << (threadIdx.x & 31 & -team);
}
// Between a team's accesses to its sample's row in global memory: the leader
// writes, every lane reads, and each waits for the others in between (a shuffle
// does not order memory).
template <bool TEAM>
__device__ __forceinline__ void team_sync(unsigned team) {
    if (TEAM) __syncwarp(team_lanes(team));
}
template <bool TEAM>
__device__ __forceinline__ bool team_leads(unsigned team) {
    return !TEAM || (threadIdx.x & (team - 1)) == 0;
}

// Shared-memory work area of one thread.
struct Work {
    Il<double> x;   // current iterate [n]
    Il<double> v;   // FP64: RHS / new iterate [n];  MIXED: residual F [n]
    Il<double> A;   // FP64 matrix [n*n]               (PREC FP64)
    Il<float> J;    // FP32 Jacobian [n*n]             (PREC MIXED)
    Il<float> d;    // FP32 RHS / step [n]             (PREC MIXED)
    int team = 1;   // lanes that hold this sample, each in its own work area
};

template <int PREC>
__host__ __device__ inline size_t work_bytes_per_thread(int n) {
    if (PREC == SP_PREC_FP64) return (size_t)(2 * n + n * n) * 8;
    // doubles first (x, F), then floats (J, d): 8-byte alignment preserved
    return (size_t)(2 * n) * 8 + (size_t)(n * n + n) * 4;
}

template <int PREC>
__device__ inline Work make_work(unsigned char* smem, int n, int bs, int tid) {
    Work w;
    double* dp = reinterpret_cast<double*>(smem);
    w.x = Il<double>{dp + tid, bs};
    w.v = Il<double>{dp + (size_t)n * bs + tid, bs};
    if (PREC == SP_PREC_FP64) {
        w.A = Il<double>{dp + (size_t)2 * n * bs + tid, bs};
        w.J = Il<float>{nullptr, bs};
        w.d = Il<float>{nullptr, bs};
    } else {
        float* fp = reinterpret_cast<float*>(dp + (size_t)2 * n * bs);
        w.A = Il<double>{nullptr, bs};
        w.J = Il<float>{fp + tid, bs};
        w.d = Il<float>{fp + (size_t)n * n * bs + tid, bs};
    }
    return w;
}

enum NrResultCode { NR_CONVERGED = 0, NR_MAXITER = 1, NR_SINGULAR = 2 };

// check_convergence (newton.rs:134-159) for old x and new xn.
__device__ inline bool step_ok(double old, double nw, double reltol, double abstol) {
    double delta = fabs(nw - old);
    double tol = reltol * fmax(fabs(nw), fabs(old)) + abstol;
    return !(delta > tol);
}

// One solve_newton_raphson from w.x; w.x holds the last iterate on return.
template <int PREC, bool TEAM = false, class DV>
__device__ inline int newton_run(const DevCircuit& c, const DV& dv, size_t s,
                                 const sp_newton_config& cfg, int mode, double aux, Work& w,
                                 int& iters) {
    const int n = c.n;
    const int nn = c.num_nodes;
    for (int it = 0; it < cfg.max_iterations; ++it) {
        if (PREC == SP_PREC_FP64) {
            for (int i = 0; i < n * n; ++i) w.A[i] = 0.0;
            for (int i = 0; i < n; ++i) w.v[i] = 0.0;
            auto k = make_sink<TEAM, PlainSink>(w.team, team_lanes(w.team), w.A, w.v, w.x, n);
            stamp_all(c, dv, s, k, mode, aux);
            if (!lu_solve_fp64(n, w.A, w.v)) {
                iters = it + 1;
                return NR_SINGULAR;
            }
            bool conv = true;
            for (int i = 0; i < n; ++i) {
                double xo = w.x[i], xn = w.v[i];
                conv = conv && step_ok(xo, xn, cfg.v_reltol, i < nn ? cfg.v_abstol : cfg.i_abstol);
                w.x[i] = xn;
            }
            if (conv) {
                iters = it + 1;
                return NR_CONVERGED;
            }
        } else {
            for (int i = 0; i < n * n; ++i) w.J[i] = 0.0f;
            for (int i = 0; i < n; ++i) w.v[i] = 0.0;
            auto k = make_sink<TEAM, MixedSink>(w.team, team_lanes(w.team), w.J, w.v, w.x, n);
            stamp_all(c, dv, s, k, mode, aux);
            for (int i = 0; i < n; ++i) w.d[i] = (float)(-w.v[i]);
            if (!lu_solve_fp32(n, w.J, w.d)) {
                iters = it + 1;
                return NR_SINGULAR;
            }
            bool conv = true;
            for (int i = 0; i < n; ++i) {
                double xo = w.x[i];
                double xn = xo + (double)w.d[i];
                conv = conv && step_ok(xo, xn, cfg.v_reltol, i < nn ? cfg.v_abstol : cfg.i_abstol);
                w.x[i] = xn;
            }
            if (conv) {
                iters = it + 1;
                return NR_CONVERGED;
            }
        }
    }
    iters = cfg.max_iterations;
    return NR_MAXITER;
}

// step_ok with its comparisons on the integer pipe, for finite values.
__device__ inline bool step_ok_int(double old, double nw, double reltol, double abstol) {
    const unsigned long long d = abs_bits(nw - old), a = abs_bits(nw), o = abs_bits(old);
    const double tol = reltol * __longlong_as_double((long long)(a > o ? a : o)) + abstol;
    return !((long long)d > __double_as_longlong(tol));
}

// newton_run of a whole warp with the solve above: every lane takes part until
// the last one is done (active false: a lane without a sample, which follows
// along on another's data).  *plain as in lu_solve_warp, cleared too where a
// start point is not finite; the caller then repeats the lane with newton_run.
template <int PREC, bool TEAM>
__device__ inline int newton_run_warp(const DevCircuit& c, const SoA& dv, size_t s, const sp_newton_config& cfg, Work& w,
                                      int& iters, bool active, bool* plain) {
    const int n = c.n, nn = c.num_nodes, lane = threadIdx.x & 31;
    const bool tols = cfg.v_reltol >= 0.0 && cfg.v_abstol >= 0.0 && cfg.i_abstol >= 0.0 && cfg.v_reltol < 1e150 &&
                      cfg.v_abstol < 1e150 && cfg.i_abstol < 1e150;
    int code = NR_MAXITER;
    iters = cfg.max_iterations;
    if (!tols) *plain = false;  // tolerances that bit patterns do not order
    for (int i = 0; i < n; ++i) *plain = *plain && finite_bits((double)w.x[i]);
    bool run = active && *plain;
    for (int it = 0; it < cfg.max_iterations && __any_sync(0xffffffffu, run); ++it) {
        bool ok, conv = true;
        if (PREC == SP_PREC_FP64) {
            for (int i = 0; i < n * n; ++i) w.A[i] = 0.0;
            for (int i = 0; i < n; ++i) w.v[i] = 0.0;
            auto k = make_sink<TEAM, PlainSinkRec>(w.team, 0xffffffffu, w.A, w.v, w.x, n, lane);
            stamp_all(c, dv, s, k, STAMP_PLAIN, 0.0);
            __syncwarp();
            ok = lu_solve_warp<double>(n, lane, w.A, w.v, k.rows, plain);
        } else {
            for (int i = 0; i < n * n; ++i) w.J[i] = 0.0f;
            for (int i = 0; i < n; ++i) w.v[i] = 0.0;
            auto k = make_sink<TEAM, MixedSinkRec>(w.team, 0xffffffffu, w.J, w.v, w.x, n, lane);
            stamp_all(c, dv, s, k, STAMP_PLAIN, 0.0);
            __syncwarp();
            for (int i = 0; i < n; ++i) w.d[i] = (float)(-w.v[i]);
            ok = lu_solve_warp<float>(n, lane, w.J, w.d, k.rows, plain);
        }
        if (run && !ok && *plain) {
            iters = it + 1;
            code = NR_SINGULAR;
            run = false;
        }
        if (!*plain) run = false;
        for (int i = 0; i < n; ++i) {
            const double xo = w.x[i];
            const double xn = PREC == SP_PREC_FP64 ? w.v[i] : xo + (double)w.d[i];
            conv = conv && step_ok_int(xo, xn, cfg.v_reltol, i < nn ? cfg.v_abstol : cfg.i_abstol);
            if (run) w.x[i] = xn;
        }
        if (run && conv) {
            iters = it + 1;
            code = NR_CONVERGED;
            run = false;
        }
    }
    return code;
}

// max_i<num_nodes |F_i| of the FP64 KCL residual at w.x (uses w.v as scratch).
template <bool TEAM = false, class DV>
__device__ inline double kcl_residual(const DevCircuit& c, const DV& dv, size_t s, Work& w) {
    for (int i = 0; i < c.n; ++i) w.v[i] = 0.0;
    auto k = make_sink<TEAM, ResidSink>(w.team, team_lanes(w.team), w.v, w.x);
    stamp_all(c, dv, s, k, STAMP_PLAIN, 0.0);
    double r = 0.0;
    for (int i = 0; i < c.num_nodes; ++i) r = fmax(r, fabs(w.v[i]));
    return r;
}

struct NewtonLaunch {
    DevCircuit c;
    sp_newton_config cfg;
    SoA dv;                 // derived constants [num_derived][stride]
    uint64_t count;         // samples in this call
    const double* x0;       // [count][n] warm starts or nullptr
    double* x;              // [count][n] output
    int32_t* iters;         // [count]
    uint8_t* status;        // [count]
    double* resid;          // [count] or nullptr
    uint32_t* fail_list;    // [count]
    unsigned int* fail_count;
    unsigned long long* work_next = nullptr;  // zeroed work counter of the persistent kernels
    // learned linear warm start evaluated by the topology-specialised kernel
    // (x0 == nullptr): x0[k] = lin_io[2 nin + k] + sum_j lin[k][j] (p[lin_slots[j]] - lin_io[j])
    // with p the sample's parameters at lin_params[slot * lin_pstride + s]
    const double* lin_params = nullptr;
    uint64_t lin_pstride = 0;
    const float* lin = nullptr;
    const float* lin_io = nullptr;
    const int* lin_slots = nullptr;
    int lin_nin = 0;
    // host copies of lin, lin_io and lin_slots (the specialised kernel takes the
    // linear term as a launch parameter when its inputs allow)
    const float* lin_host = nullptr;
    const float* lin_io_host = nullptr;
    const int* lin_slots_host = nullptr;
    // per-sample parameters [slot][params_stride] for the specialised kernel's
    // parameters mode, which writes the FP64 derived constants of the samples it
    // lists for the fallback into derived_out (same layout as dv)
    const double* params = nullptr;
    uint64_t params_stride = 0;
    double* derived_out = nullptr;
    // per-block moments of the specialised kernel (one sample per thread), [n][grid]
    sp_moments* moments_partial = nullptr;
    // FP32 drawn parameters of the specialised kernel ([slot][params_stride], then
    // params is not read), and what the fallback needs to draw its samples in FP64
    const float* params32 = nullptr;
    RedrawArgs redraw;
    // lanes per sample (a power of two): the primary kernel's, and the most the
    // fallback takes where its list leaves lanes idle
    int team = 1, fallback_team = 1;
    // iteration limit of the specialised kernel's cold restart of a sample
    // whose warm start missed (the full limit; cfg may hold the warm cap)
    int cold_max_iterations = 0;
};

__device__ inline void load_start(const NewtonLaunch& L, size_t s, Work& w, bool warm) {
    const int n = L.c.n;
    if (warm) {
        for (int i = 0; i < n; ++i) w.x[i] = L.x0[s * n + i];
    } else if (L.c.nodeset) {
        for (int i = 0; i < n; ++i) w.x[i] = L.c.nodeset[i];
    } else {
        for (int i = 0; i < n; ++i) w.x[i] = 0.0;
    }
}

__device__ inline uint8_t finish_status(int code, const Work& w, int n) {
    for (int i = 0; i < n; ++i)
        if (!isfinite(w.x[i])) return SP_ST_NONFINITE;
    if (code == NR_CONVERGED) return SP_ST_CONVERGED;
    return code == NR_SINGULAR ? SP_ST_SINGULAR : SP_ST_FAILED;
}

// The __global__ templates below are instantiated by two translation units
// compiled with different FMA settings; each unit picks its own namespace
// (SP_KERNEL_NS) so that the two instantiations are distinct kernels.
#ifndef SP_KERNEL_NS
#define SP_KERNEL_NS kdefault
#endif
namespace SP_KERNEL_NS {

// Phase 1: Newton from the warm start (or the circuit's nodeset, or zero)
// for every sample; misses go to the fallback list.
template <int PREC, bool TEAM = false>
__global__ void newton_primary_kernel(NewtonLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_wait();
    pdl_trigger();
    const uint64_t s = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / (TEAM ? (unsigned)L.team : 1u);
    Work w = make_work<PREC>(smem, L.c.n, blockDim.x, threadIdx.x);
    w.team = TEAM ? L.team : 1;
    const int n = L.c.n;
    const bool warm = L.x0 != nullptr;
    int it = 0, code;
#ifdef SP_EXACT_UNIT
    // a skipped product with a zero could leave a -0 where the reference has +0
    if (s >= L.count) return;
    load_start(L, s, w, warm);
    code = newton_run<PREC, TEAM>(L.c, L.dv, s, L.cfg, STAMP_PLAIN, 0.0, w, it);
#else
    const bool active = s < L.count;
    const uint64_t sd = active ? s : L.count - 1;
    // the sample's constants on their way to L1 together (each stamp waits for its own)
    for (int k = 0; k < L.c.num_derived; ++k)
        asm volatile("prefetch.global.L1 [%0];" ::"l"(L.dv.p + (size_t)k * L.dv.stride + sd));
    bool plain = true;
    load_start(L, sd, w, warm);
    code = newton_run_warp<PREC, TEAM>(L.c, L.dv, sd, L.cfg, w, it, active, &plain);
    if (!active) return;
    if (!plain) {  // by single lanes: the teams of a warp part here
        load_start(L, s, w, warm);
        code = newton_run<PREC>(L.c, L.dv, s, L.cfg, STAMP_PLAIN, 0.0, w, it);
    }
#endif
    const bool lead = !TEAM || (threadIdx.x & (L.team - 1)) == 0;  // the others hold the same values
    uint8_t st = finish_status(code, w, n) | (warm ? SP_ST_FLAG_WARM : 0);
    if (lead)
        for (int i = 0; i < n; ++i) L.x[s * n + i] = w.x[i];
    if (lead && L.iters) L.iters[s] = it;
    bool need_fallback = (st & SP_ST_MASK) != SP_ST_CONVERGED &&
                         (warm || (L.cfg.fallback & (SP_FALLBACK_GMIN | SP_FALLBACK_SOURCE)));
    if (need_fallback) {
        if (lead) {
            unsigned int slot = atomicAdd(L.fail_count, 1u);
            L.fail_list[slot] = (uint32_t)s;
        }
    } else if (L.resid) {
        const double r = kcl_residual<TEAM>(L.c, L.dv, s, w);
        if (lead) L.resid[s] = r;
    }
    if (lead && L.status) L.status[s] = st;
}

}  // namespace SP_KERNEL_NS

// A sample's row of unknowns, written by its team's leader once every lane has
// read what was there, and there for every lane on return.
template <bool TEAM, class F>
__device__ __forceinline__ void put_row(unsigned team, int n, double* row, F value) {
    team_sync<TEAM>(team);
    if (team_leads<TEAM>(team))
        for (int i = 0; i < n; ++i) row[i] = value(i);
    team_sync<TEAM>(team);
}

// gmin stepping (newton.rs:373-459).  The level solution lives in the
// output row (global), the trial iterate in shared memory.  A failed attempt
// is repeated by the reference with the identical initial guess and stamper,
// so its outcome repeats; those repeats are accounted without recomputation.
template <int PREC, bool TEAM, class DV>
__device__ inline int gmin_stepping(const NewtonLaunch& L, const DV& dv, size_t s, Work& w, int& total) {
    const int n = L.c.n;
    const sp_newton_config& cfg = L.cfg;
    double* sol = L.x + s * n;
    put_row<TEAM>(w.team, n, sol, [](int) { return 0.0; });
    double g = cfg.gmin_initial;
    int levels = 0;
    while (g >= cfg.gmin_final * 0.99 && levels < 4096) {
        ++levels;
        for (int i = 0; i < n; ++i) w.x[i] = sol[i];
        int it = 0;
        int code = newton_run<PREC, TEAM>(L.c, dv, s, cfg, STAMP_GMIN, g, w, it);
        total += it;
        if (code == NR_SINGULAR) return NR_SINGULAR;
        if (code != NR_CONVERGED) {
            total += (cfg.gmin_max_attempts - 1) * it;
            return NR_MAXITER;
        }
        put_row<TEAM>(w.team, n, sol, [&](int i) { return w.x[i]; });
        if (g <= cfg.gmin_final) break;
        g /= cfg.gmin_reduction;
        if (g < cfg.gmin_final) g = cfg.gmin_final;
    }
    return NR_CONVERGED;
}

// source stepping (newton.rs:261-356).
template <int PREC, bool TEAM, class DV>
__device__ inline int source_stepping(const NewtonLaunch& L, const DV& dv, size_t s, Work& w, int& total) {
    const int n = L.c.n;
    const sp_newton_config& cfg = L.cfg;
    double* sol = L.x + s * n;
    put_row<TEAM>(w.team, n, sol, [](int) { return 0.0; });
    double factor = cfg.src_initial;
    double step = cfg.src_step;
    int guard = 0;
    while (factor <= 1.0 + 1e-9 && guard < 100000) {
        ++guard;
        double cur = fmin(factor, 1.0);
        for (int i = 0; i < n; ++i) w.x[i] = sol[i];
        int it = 0;
        int code = newton_run<PREC, TEAM>(L.c, dv, s, cfg, STAMP_SCALED, cur, w, it);
        total += it;
        if (code == NR_SINGULAR) return NR_SINGULAR;
        if (code != NR_CONVERGED) {
            total += (cfg.src_max_attempts - 1) * it;
            if (step > cfg.src_min_step) {
                step /= 2.0;
                factor -= step;
                continue;
            }
            return NR_MAXITER;
        }
        put_row<TEAM>(w.team, n, sol, [&](int i) { return w.x[i]; });
        if (fabs(cur - 1.0) < 1e-9) break;
        factor += step;
        if (step < cfg.src_step) step = fmin(step * 1.5, cfg.src_step);
    }
    return NR_CONVERGED;
}

namespace SP_KERNEL_NS {

// The fallback chain of one sample, held by `team` lanes.  All of them take the
// same branches: what decides one comes from values that each has computed
// alike, or from the sample's row, which changes only in put_row.
template <int PREC, bool TEAM, class DV>
__device__ inline void fallback_sample(const NewtonLaunch& L, const DV& dv, size_t s, Work& w, unsigned team) {
    const int n = L.c.n;
    const bool warm = L.x0 != nullptr || L.lin != nullptr;  // listed samples started warm
    const bool lead = team_leads<TEAM>(team);
    w.team = (int)team;
    if (L.redraw.derived) redraw_sample(L.c, L.redraw, L.dv.stride, s);
    int total = L.iters ? L.iters[s] : 0;
    uint8_t flags = warm ? SP_ST_FLAG_WARM : 0;
    // A stage succeeds only if it converged with a finite iterate (the
    // reference's convergence test passes NaN iterates).
    auto ok = [&](int code) {
        if (code != NR_CONVERGED) return false;
        for (int i = 0; i < n; ++i)
            if (!isfinite(L.x[s * n + i])) return false;
        return true;
    };
    int code = NR_MAXITER;
    // the specialised kernel has already restarted this sample cold (status
    // flag), so the chain continues with gmin stepping
    const bool cold_done = warm && L.status && (L.status[s] & SP_ST_FLAG_COLD);
    team_sync<TEAM>(team);  // read before the leader writes them
    if (cold_done) flags |= SP_ST_FLAG_COLD;
    if (warm && !cold_done) {
        flags |= SP_ST_FLAG_COLD;
        load_start(L, s, w, false);
        int it = 0;
        code = newton_run<PREC, TEAM>(L.c, dv, s, L.cfg, STAMP_PLAIN, 0.0, w, it);
        total += it;
        put_row<TEAM>(team, n, L.x + s * n, [&](int i) { return w.x[i]; });
    }
    if (!ok(code) && (L.cfg.fallback & SP_FALLBACK_GMIN)) {
        flags |= SP_ST_FLAG_GMIN;
        code = gmin_stepping<PREC, TEAM>(L, dv, s, w, total);
    }
    if (!ok(code) && (L.cfg.fallback & SP_FALLBACK_SOURCE)) {
        flags |= SP_ST_FLAG_SOURCE;
        code = source_stepping<PREC, TEAM>(L, dv, s, w, total);
    }
    for (int i = 0; i < n; ++i) w.x[i] = L.x[s * n + i];
    uint8_t st = finish_status(code, w, n) | flags;
    const double res = L.resid ? kcl_residual<TEAM>(L.c, dv, s, w) : 0.0;
    if (lead && L.iters) L.iters[s] = total;
    if (lead && L.status) L.status[s] = st;
    if (lead && L.resid) L.resid[s] = res;
}

// Phase 2: the fallback chain for the samples phase 1 missed (grid-stride
// over the miss list, whose length is only known on the device; one-warp blocks).
template <int PREC, bool TEAM = false>
__global__ void newton_fallback_kernel(NewtonLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    pdl_wait();
    pdl_trigger();
    Work w = make_work<PREC>(smem, L.c.n, blockDim.x, threadIdx.x);
    const unsigned int misses = *L.fail_count;
    const SoAOwn dv{L.dv.p, L.dv.stride};
    // A list of at most a sample per block: a team of the block's lanes takes it,
    // every one of them with its data.  Longer lists go to single lanes: teams of
    // one warp part at the first stage of different length, and every shuffle and
    // barrier of theirs then runs once per team (608 chains of eight devices, all
    // failing: 447 ms with several teams in a warp, or teams of one lane; 112 so).
    if (TEAM && misses <= gridDim.x) {
        if (blockIdx.x < misses && threadIdx.x < (unsigned)L.fallback_team)
            fallback_sample<PREC, true>(L, dv, L.fail_list[blockIdx.x], w, (unsigned)L.fallback_team);
        return;
    }
    // neighbours in the list go to different blocks: chains differ in length at
    // every level, and lanes of one warp wait for each other there
    for (unsigned int j = threadIdx.x * gridDim.x + blockIdx.x; j < misses; j += gridDim.x * blockDim.x)
        fallback_sample<PREC, false>(L, dv, L.fail_list[j], w, 1);
}

}  // namespace SP_KERNEL_NS
}  // namespace sp
