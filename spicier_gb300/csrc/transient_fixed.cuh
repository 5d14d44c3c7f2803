// Batched fixed-step linear transients (solve_transient, solver.rs:41-252),
// one thread per sample, after the DC operating point of the same samples.
//
// The circuit is linear and the step fixed, so the matrix of a stage (R, V
// and the companion conductances of companion.rs: BE, TRAP, or the TR-BDF2
// pair of stages) does not change from step to step: it is stamped and
// factorised once per sample by the nalgebra-order LU of the DC path, and a
// step builds its right-hand side (sources at t = step h in element order,
// then the capacitors' and the inductors' companion currents), applies the
// factor's row order and substitutes.  Every right-hand side entry and unknown
// goes through the operations of the reference's per-step solve in the same
// order, so in the exact translation unit (no FMA) a run is bit-identical to
// the oracle's linear_transient; the states follow the reference's update
// rules, including its TR-BDF2 updates as written.  Unknowns: nodes + V-source
// currents (inductors carry no branch variable in the transient MNA).
//
// What bounds it: an FP64 instruction takes a warp 64 cycles of its SM
// quarter's pipe, and 16,384 samples are less than one warp per quarter, so a
// step costs its FP64 instruction count.  Besides the factorisation (2/3 n^3
// per stage), the step leaves out the divisions by h (companion conductances
// are kept), the substitution's divisions (reciprocals of the diagonal are
// kept, with one correction step) and, outside the exact unit, the factor's
// zeros.  16,384 samples of a 9-unknown RLC network, 150 trapezoidal steps:
// 6.2 -> 1.5 ms (TR-BDF2 holds two factors a sample; runs of one or two steps lose a
// little: 16,384 samples of 10 unknowns, 2 steps, 0.42 ms instead of 0.36).
#pragma once
#include <math_constants.h>

#include "newton_dense.cuh"

namespace sp {

// An element that enters a step's right-hand side: ref is the pulse of a
// source, -1 - slot of a constant one's value, or the slot of C or L.
struct TransientEl {
    int n0, n1, ref, kind;
};

struct TransientLaunch {
    DevCircuit c;
    const TransientEl* els;    // V and I sources, then capacitors, then inductors, each in element order
    int num_src, num_caps, num_inds, num_pulses;
    const double* params;      // [count][np] (the DC pass's drawn parameters)
    int np;
    const double* x_dc;        // [count][n_dc]
    uint64_t count;
    int method;                // 0 BE, 1 TRAP, 2 TR-BDF2
    double h, tstop;
    long steps;
    int nt;                    // transient unknowns
    int keep;                  // companion conductances kept per sample (they fit)
    int wave_steps;            // steps whose source waveforms are tabulated at a time (0: none are)
    int probe_idx;
    double* x;                 // [count][nt]
    double* probe;             // [count][steps + 1] or nullptr
    uint8_t* status;           // in: DC status; out: transient status
};

// Shared doubles per thread: the factors (two stages in TR-BDF2) with their
// diagonal's reciprocals and row orders, right-hand side and solution, and per
// reactive element v, i (and the value two points back), and what is kept of
// its conductances.
__host__ __device__ inline size_t transient_words(int nt, int reactive, int method, bool keep) {
    const size_t f = method == 2 ? 2 : 1, n = nt;
    return f * (n * n + n + (n + 1) / 2) + 2 * n + (size_t)reactive * ((method == 2 ? 3 : 2) + (keep ? (method == 2 ? 3 : 1) : 0));
}
// Shared doubles per warp: the waveform table and the factors' patterns.
__host__ __device__ inline size_t transient_warp_words(int nt, int num_pulses, int wave_steps, int method) {
    return (size_t)num_pulses * wave_steps + (method == 2 ? 2 : 1) * (size_t)nt;
}

#ifdef SP_KERNEL_NS
namespace SP_KERNEL_NS {

#ifdef SP_EXACT_UNIT
constexpr bool kTranExact = true;
#else
constexpr bool kTranExact = false;
#endif

__device__ inline double tr_pulse(const sp_pulse& p, double t) {
    if (t < p.td) return p.v1;
    const double t_rel = p.per > 0.0 ? fmod(t - p.td, p.per) : t - p.td;
    if (t_rel < p.tr) return p.v1 + (p.v2 - p.v1) * t_rel / p.tr;
    if (t_rel < p.tr + p.pw) return p.v2;
    if (t_rel < p.tr + p.pw + p.tf) return p.v2 - (p.v2 - p.v1) * (t_rel - p.tr - p.pw) / p.tf;
    return p.v1;
}

__global__ void transient_fixed_kernel(TransientLaunch L) {
    extern __shared__ __align__(16) double tsm[];
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const DevCircuit& c = L.c;
    const int nt = L.nt, nn = c.num_nodes, bs = blockDim.x, lane = threadIdx.x & 31;
    const unsigned wmask = bs >= 32 ? 0xffffffffu : (1u << bs) - 1u;  // the lanes of this warp (bs: a power of two)
    const int stages = L.method == 2 ? 2 : 1, nr = L.num_caps + L.num_inds;
    const bool bdf = L.method == 2;
    // this warp's region, then the interleaved per-thread arrays
    const int warps = (bs + 31) / 32;
    double* wave = tsm + (size_t)(threadIdx.x >> 5) * transient_warp_words(nt, L.num_pulses, L.wave_steps, L.method);
    unsigned* pat = reinterpret_cast<unsigned*>(wave + (size_t)L.num_pulses * L.wave_steps);  // [stage][L rows, U rows][nt]
    double* base = tsm + (size_t)warps * transient_warp_words(nt, L.num_pulses, L.wave_steps, L.method) + threadIdx.x;
    auto take = [&](size_t words) {
        const Il<double> a{base, bs};
        base += words * bs;
        return a;
    };
    Il<double> A[2], rd[2];
    Il<int> at[2];  // at[q][r]: the position of equation r in the factor's row order
    for (int q = 0; q < stages; ++q) {
        A[q] = take((size_t)nt * nt);
        rd[q] = take(nt);
        at[q] = Il<int>{reinterpret_cast<int*>(base - threadIdx.x) + threadIdx.x, bs};
        base += (size_t)((nt + 1) / 2) * bs;
    }
    const Il<double> b = take(nt), xs = take(nt), v = take(nr), cur = take(nr), pp = take(bdf ? nr : 0);
    const Il<double> kept = take(L.keep ? (size_t)nr * (bdf ? 3 : 1) : 0);
    const bool live = s < L.count && (L.status[s < L.count ? s : 0] & SP_ST_MASK) == SP_ST_CONVERGED;
    const uint64_t si = s < L.count ? s : 0;
    auto P = [&](int slot) { return L.params[si * L.np + slot]; };
    double* xo = L.x + si * nt;
    if (s < L.count && !live)
        for (int i = 0; i < nt; ++i) xo[i] = CUDART_NAN;  // keeps the DC status
    const TransientEl* els = L.els;
    const TransientEl* react = els + L.num_src;
    const int ndc = nn + c.num_branches;
    const double* dc = L.x_dc + si * ndc;
    auto nv = [&](const double* x, int i) { return i >= 0 ? x[i] : 0.0; };
    auto nvi = [&](Il<double> x, int i) { return i >= 0 ? x[i] : 0.0; };
    const double h = L.h, gamma = 2.0 - 1.4142135623730951;
    const double hg = bdf ? gamma * h : h;
    const double h2 = (1.0 - gamma) * h, h1 = gamma * h, rho = h2 / h1, denom = 1.0 + 2.0 * rho;
    const double a1 = (1.0 + rho) * (1.0 + rho) / denom, a2 = -rho * rho / denom, b0 = (1.0 + rho) / denom;
    const double alpha = (1.0 - gamma) / (gamma * (2.0 - gamma));
    // companion conductance of reactive element j: kind 0 BE, 1 TRAP (of step hg), 2 the BDF2 stage;
    // kind 3: C / h or h / L of the TR-BDF2 state update
    auto conductance = [&](int j, int kind) {
        const double val = P(react[j].ref);
        if (j < L.num_caps) return kind == 0 || kind == 3 ? val / h : kind == 1 ? 2.0 * val / hg : val / (b0 * h2);
        return kind == 0 || kind == 3 ? h / val : kind == 1 ? hg / (2.0 * val) : b0 * h2 / val;
    };
    auto geq = [&](int j, int kind) {
        return L.keep ? kept[bdf ? 3 * j + kind - 1 : j] : conductance(j, kind);
    };
    const int first_kind = bdf ? 1 : L.method;

    // states and solution from the DC operating point, matrices and factors
    uint8_t status = SP_ST_CONVERGED;
    if (live) {
        int kv = 0, kc = 0, kl = 0;
        for (int e = 0; e < c.num_elements; ++e) {
            const sp_element& el = c.el[e];
            if (el.kind == SP_EL_C || el.kind == SP_EL_L) {
                const int j = el.kind == SP_EL_C ? kc++ : L.num_caps + kl++;
                v[j] = nv(dc, el.node[0]) - nv(dc, el.node[1]);
                cur[j] = el.kind == SP_EL_L ? dc[nn + el.branch] : 0.0;
                if (bdf) pp[j] = 0.0;
            } else if (el.kind == SP_EL_V) {
                xs[nn + kv] = dc[nn + el.branch];
                ++kv;
            }
        }
        for (int i = 0; i < nn; ++i) xs[i] = dc[i];
        if (L.keep)
            for (int j = 0; j < nr; ++j)
                for (int k = 0; k < (bdf ? 3 : 1); ++k) kept[bdf ? 3 * j + k : j] = conductance(j, bdf ? k + 1 : first_kind);
    }
    for (int q = 0; q < stages; ++q) {
        Il<double> M = A[q];
        if (live) {
            for (int i = 0; i < nt * nt; ++i) M[i] = 0.0;
            for (int i = 0; i < nt; ++i) b[i] = (double)i;  // the rows' order, permuted with the factor
            auto add = [&](int r, int col, double g) { M[col * nt + r] += g; };
            auto cond = [&](int i, int j, double g) {
                if (i >= 0) add(i, i, g);
                if (j >= 0) add(j, j, g);
                if (i >= 0 && j >= 0) {
                    add(i, j, -g);
                    add(j, i, -g);
                }
            };
            int kv = 0;
            for (int e = 0; e < c.num_elements; ++e) {
                const sp_element& el = c.el[e];
                const int n0 = el.node[0], n1 = el.node[1];
                if (el.kind == SP_EL_R) {
                    cond(n0, n1, 1.0 / P(el.field[0]));
                } else if (el.kind == SP_EL_V) {
                    const int row = nn + kv++;
                    if (n0 >= 0) {
                        add(n0, row, 1.0);
                        add(row, n0, 1.0);
                    }
                    if (n1 >= 0) {
                        add(n1, row, -1.0);
                        add(row, n1, -1.0);
                    }
                }
            }
            for (int j = 0; j < nr; ++j) cond(react[j].n0, react[j].n1, geq(j, q ? 2 : first_kind));
            lu_factor_fp64(nt, M, b);
            for (int i = 0; i < nt; ++i) {
                at[q][(int)b[i]] = i;
                const double d = M[i * nt + i];
                if (d == 0.0) status = SP_ST_SINGULAR;
                rd[q][i] = mid_range(d) ? 1.0 / d : 0.0;  // kept where the correction step below holds
            }
        }
        __syncwarp(wmask);
        // the warp's pattern: entries that are nonzero in some sample (all of them in the exact unit,
        // where a product with a zero may still turn a -0 into +0)
        for (int i = 0; i < nt; ++i) {
            unsigned lo = 0, up = 0;
            if (live)
                for (int k = 0; k < nt; ++k)
                    if (k != i && (kTranExact || M[k * nt + i] != 0.0)) (k < i ? lo : up) |= 1u << k;
            lo = __reduce_or_sync(wmask, lo);
            up = __reduce_or_sync(wmask, up);
            if (lane == 0) pat[(2 * q) * nt + i] = lo, pat[(2 * q + 1) * nt + i] = up;
        }
    }
    __syncwarp(wmask);

    double* pr = L.probe && L.probe_idx >= 0 && s < L.count ? L.probe + s * (L.steps + 1) : nullptr;
    if (pr && live) pr[0] = xs[L.probe_idx];
    if (live && L.steps < 1) status = SP_ST_CONVERGED;
    const bool run = live && status == SP_ST_CONVERGED;
    auto inject = [&](int q, int i, double add) {
        if (i >= 0) {
            const int p = at[q][i];
            b[p] += add;
        }
    };
    // right-hand side at time t of a stage, in the factor's row order; ki: waveform table row
    auto rhs = [&](int q, int kind, int ki, double t) {
        for (int i = 0; i < nt; ++i) b[i] = 0.0;
        int row = nn;
        for (int k = 0; k < L.num_src; ++k) {
            const TransientEl el = els[k];
            const double val = el.ref < 0 ? P(-1 - el.ref)
                                          : L.wave_steps ? wave[(size_t)ki * L.num_pulses + el.ref] : tr_pulse(c.pulses[el.ref], t);
            if (el.kind == SP_EL_V) {
                b[at[q][row++]] = val;
            } else {
                inject(q, el.n0, -val);
                inject(q, el.n1, val);
            }
        }
        for (int j = 0; j < nr; ++j) {
            const TransientEl el = react[j];
            const double g = kind == 2 && j >= L.num_caps ? 0.0 : geq(j, kind);
            double ieq;
            if (j < L.num_caps) {
                ieq = kind == 0 ? g * v[j] : kind == 1 ? g * v[j] + cur[j] : g * (a1 * v[j] + a2 * pp[j]);
                inject(q, el.n1, -ieq);
                inject(q, el.n0, ieq);
            } else {
                ieq = kind == 0 ? cur[j] : kind == 1 ? cur[j] + g * v[j] : a1 * cur[j] + a2 * pp[j];
                inject(q, el.n0, -ieq);
                inject(q, el.n1, ieq);
            }
        }
    };
    // substitutions; the solution replaces b.  Row by row: each unknown takes its
    // updates in the order of the column-oriented solve, from a register.
    auto substitute = [&](int q) {
        const Il<double> M = A[q];
        bool fin = true;
        for (int i = 0; i < nt; ++i) {
            double acc = b[i];
            unsigned m = pat[(2 * q) * nt + i];
            if (!fin) m = (1u << i) - 1u;  // a non-finite entry reaches every row, as in the dense solve
            while (m) {
                const int k = __ffs(m) - 1;
                m &= m - 1;
                acc = -b[k] * M[k * nt + i] + acc;
            }
            if (!kTranExact) fin = fin && finite_bits(acc);
            b[i] = acc;
        }
        for (int i = nt - 1; i >= 0; --i) {
            double acc = b[i];
            unsigned m = pat[(2 * q + 1) * nt + i];
            if (!fin) m = nt >= 32 ? ~((2u << i) - 1u) : ((1u << nt) - 1u) & ~((2u << i) - 1u);
            while (m) {
                const int k = 31 - __clz(m);
                m ^= 1u << k;
                acc = -b[k] * M[k * nt + i] + acc;
            }
            // acc / d as IEEE division gives it, by one step from the reciprocal where
            // nothing leaves the normal range (and for +0; a -0 would lose its sign).
            // With significands a, b in [1, 2) and u an ulp of a / b: r = (1 + e) / b,
            // |e| <= b 2^-54, so acc r is less than u off, and where a / b is near the
            // midpoint of two doubles the first product is one of the two, its remainder
            // exact, and the corrected value at most |e| (u / 2 + t) off, t the distance
            // to the midpoint.  t >= 2^-53 u / b is more than that, as b^2 < 4 - 2^-51.
            const double d = M[i * nt + i], r = rd[q][i];
            double x = acc * r;
            x = fma(fma(-d, x, acc), r, x);
            const long long ab = __double_as_longlong(acc), rb = __double_as_longlong(r);
            if (kTranExact || rb == 0 || !(ab == 0 || mid_range(acc))) x = acc / d;
            if (!kTranExact) fin = fin && finite_bits(x);
            b[i] = x;
        }
    };
    auto across = [&](int j, Il<double> x) { return nvi(x, react[j].n0) - nvi(x, react[j].n1); };
    const int chunk = L.wave_steps ? L.wave_steps : 32;
    for (long step0 = 0; step0 < L.steps; step0 += chunk) {
        // source waveforms of the next steps, one step per lane
        __syncwarp(wmask);
        for (int k = lane; k < L.wave_steps * L.num_pulses; k += bs < 32 ? bs : 32) {
            const long step = step0 + 1 + k / L.num_pulses;
            if (step <= L.steps) wave[k] = tr_pulse(c.pulses[k % L.num_pulses], (double)step * h);
        }
        __syncwarp(wmask);
        const long last = step0 + chunk < L.steps ? step0 + chunk : L.steps;
        if (run)
            for (long step = step0 + 1; step <= last; ++step) {
                const int ki = (int)(step - 1 - step0);
                const double t = (double)step * h;
                if (bdf) {
                    rhs(0, 1, ki, t);
                    substitute(0);
                    for (int j = 0; j < nr; ++j) {
                        const double vn = across(j, b);
                        if (j < L.num_caps) {
                            pp[j] = v[j];
                            cur[j] = geq(j, 1) * (vn - v[j]) - cur[j];
                        } else {
                            pp[j] = cur[j];
                            cur[j] += geq(j, 1) * (vn + v[j]);
                        }
                        v[j] = vn;
                    }
                    rhs(1, 2, ki, t);
                    substitute(1);
                } else {
                    rhs(0, L.method, ki, t);
                    substitute(0);
                }
                for (int i = 0; i < nt; ++i) xs[i] = b[i];
                for (int j = 0; j < nr; ++j) {
                    const double vn = across(j, xs), g = geq(j, bdf ? 3 : L.method);
                    if (j < L.num_caps) {
                        if (L.method == 0) cur[j] = g * (vn - v[j]);
                        else if (L.method == 1) cur[j] = g * (vn - v[j]) - cur[j];
                        else cur[j] = g * ((1.0 + alpha) * vn - (1.0 + 2.0 * alpha) * v[j] + alpha * pp[j]);
                        if (bdf) pp[j] = v[j];
                    } else {
                        if (L.method == 0) cur[j] += g * vn;
                        else if (L.method == 1) cur[j] += g * (vn + v[j]);
                        else cur[j] += g * ((1.0 + alpha) * vn - (1.0 + 2.0 * alpha) * v[j] + alpha * v[j]);
                        if (bdf) pp[j] = cur[j];
                    }
                    v[j] = vn;
                }
                if (pr) pr[step] = xs[L.probe_idx];
            }
    }
    if (!live) return;
    if (!run && pr)
        for (long k = 1; k <= L.steps; ++k) pr[k] = CUDART_NAN;  // every step's solve is singular
    for (int i = 0; i < nt; ++i) xo[i] = xs[i];
    L.status[s] = status;
}

}  // namespace SP_KERNEL_NS
#endif  // SP_KERNEL_NS

}  // namespace sp
