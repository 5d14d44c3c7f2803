// FP64 AC sweeps on the circuit's pattern: a warp solves the complex systems of
// 32 (sample, frequency) units together.
//
// The dense solve (ac.cuh) kept n^2 + n complex doubles per unit in shared
// memory (2.5 KB for the op-amp: two warps per SM), evaluated the devices again
// at every frequency and spent eight FP64 operations on every product, most of
// them with a zero part.  Here
//
//   ac_values_kernel  evaluates each sample's devices once and stores its real
//                     entries and reactive values;
//   ac_sparse_kernel  keeps only the parts that can be nonzero, real and
//                     imaginary separately, in shared-memory slots shared by the
//                     warp's lanes: a map from (column, row) to a slot per part.
//                     Every unit of a warp has the same circuit, so the map, the
//                     fill and (nearly always) the pivots are the warp's; a row
//                     swap exchanges map entries, and only lanes that pivot
//                     differently move values.
//
// Each part takes the operations of the dense solve in its order without those
// whose product is an exact zero.  The matrix and right-hand side start from +0
// and only ever take sums, so an absent part is +0 there too, and skipping the
// addition of a zero product leaves the same bits; a probed unknown's quotient
// is formed from all its parts, which gives its zeros their signs.  Values that
// are not finite (whose product with a zero is not zero) and systems that
// outgrow the slots go to the dense kernel, as do sweeps of circuits whose
// estimated fill (ac_plan.h) makes it the faster one.
//
// Bound: the FP64 pipe (64 cycles per warp instruction of an SM quarter) and,
// with two warps per quarter, the chains between its instructions.  Op-amp,
// 8,192 samples x 81 frequencies: 19.5 -> 2.8 ms (the call with its DC points: 20.0 -> 3.2).
#pragma once
#include "ac.cuh"

namespace sp {

// Shared bytes of one warp: values, two maps, the pivots' reciprocal slots.
__host__ __device__ inline size_t ac_sparse_warp_bytes(int n, int cap) {
    const size_t map = 2 * (size_t)(n + 1) * n;
    return 256 * (size_t)cap + ((2 * map + 2 * n + 255) & ~size_t(255));
}

#ifdef SP_AC_KERNELS
__global__ void __launch_bounds__(128) ac_values_kernel(AcLaunch L) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= L.count || (L.dc_status[s] & SP_ST_MASK) != SP_ST_CONVERGED) return;
    const int n = L.c.n, bs = blockDim.x;
    double* A = reinterpret_cast<double*>(ac_smem) + threadIdx.x;
    for (int k = 0; k < n * n; ++k) A[(size_t)k * bs] = 0.0;
    ac_real_stamps(
        L, s,
        [&](int r, int c, double v) {
            if (r >= 0 && c >= 0) A[(size_t)(c * n + r) * bs] += v;
        },
        [](int) {});
    for (int k = 0; k < L.num_entries; ++k) {
        const AcEntry e = L.entries[k];
        L.values[(size_t)k * L.count + s] = A[(size_t)(e.c * n + e.r) * bs];
    }
    const double* P = L.params + s * (uint64_t)L.np;
    for (int e = 0, v = L.num_entries; e < L.c.num_elements; ++e) {
        const sp_element el = L.c.el[e];
        if (el.kind == SP_EL_C || el.kind == SP_EL_L) {
            L.values[(size_t)v++ * L.count + s] = P[el.field[0]];
        } else if (el.kind == SP_EL_BSIM3N || el.kind == SP_EL_BSIM3P) {
            double g[8];
            bsim3_ac_values(L, s, e, el, P, L.x_dc + s * (uint64_t)n, g);
            for (int k = 3; k < 8; ++k) L.values[(size_t)v++ * L.count + s] = g[k];
        }
    }
}

// The warp's state: slots and masks.  Lane c < n + 1 holds the rows of column c
// (column n: the right-hand side) that have a real / an imaginary part.
struct AcWarp {
    double* val;      // [cap][32], this lane's column
    uint16_t *mr, *mi;  // [(n + 1) n] slots of the parts, meaningful where the masks say so
    int n, lane, cap;
    unsigned rows_r, rows_i;
    int used;
    bool over, fin;

    __device__ double& at(int slot) const { return val[slot * 32]; }
    __device__ double get(const uint16_t* m, int c, int r) const { return at(m[c * n + r]); }
    __device__ void check(double v) { fin = fin && finite_bits(v); }
    // a new slot for a part of entry (r, c); the map is the warp's
    __device__ int add_slot(uint16_t* m, unsigned& rows, int c, int r) {
        if (used >= cap) over = true;
        const int s = used < cap ? used++ : cap - 1;
        if (lane == 0) m[c * n + r] = (uint16_t)s;
        if (lane == c) rows |= 1u << r;
        __syncwarp();
        return s;
    }
    // part += v, or = v in a new slot (whose part was +0)
    __device__ void acc(uint16_t* m, unsigned& rows, bool present, int c, int r, double v) {
        if (present) {
            double& d = at(m[c * n + r]);
            v = v + d;
            d = v;
        } else {
            v = v + 0.0;
            at(add_slot(m, rows, c, r)) = v;
        }
        check(v);
    }
};

__global__ void __launch_bounds__(128) ac_sparse_kernel(AcLaunch L) {
    extern __shared__ __align__(16) unsigned char ac_smem[];
    const DevCircuit& c = L.c;
    const int n = c.n, nn = c.num_nodes, lane = threadIdx.x & 31;
    unsigned char* base = ac_smem + (size_t)(threadIdx.x >> 5) * ac_sparse_warp_bytes(n, L.cap);
    AcWarp W;
    W.val = reinterpret_cast<double*>(base) + lane;
    W.mr = reinterpret_cast<uint16_t*>(base + 256 * (size_t)L.cap);
    W.mi = W.mr + (n + 1) * n;
    uint16_t* rns = W.mi + (n + 1) * n;  // [n] slot of 1 / |pivot|^2
    W.n = n;
    W.lane = lane;
    W.cap = L.cap;
    unsigned probed = 0, base_rows = 0;
    for (int k = 0; k < L.num_entries; ++k)
        if (L.entries[k].c == lane) base_rows |= 1u << L.entries[k].r;
    for (int k = 0; k < L.num_probe; ++k) probed |= 1u << L.probe[k];
    const uint64_t total = L.count * (uint64_t)L.nf;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t g = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g * 32 < total; g += warps) {
        const uint64_t u = g * 32 + lane < total ? g * 32 + lane : total - 1;
        const bool active = g * 32 + lane < total;
        uint64_t s = u / (uint64_t)L.nf;
        int f = (int)(u - s * (uint64_t)L.nf);
        const bool live = active && (L.dc_status[s] & SP_ST_MASK) == SP_ST_CONVERGED;
        double* out = L.out + u * (uint64_t)L.num_probe * 2;
        if (active && !live)
            for (int k = 0; k < 2 * L.num_probe; ++k) out[k] = CUDART_NAN;
        const unsigned any = __ballot_sync(0xffffffffu, live);
        if (!any) continue;
        {  // a lane without a unit follows along on another's, so that it pivots like it
            const int src = __ffs(any) - 1;
            const uint64_t s1 = __shfl_sync(0xffffffffu, s, src);
            const int f1 = __shfl_sync(0xffffffffu, f, src);
            if (!live) s = s1, f = f1;
        }
        // matrix: the real entries' slots are their numbers
        W.rows_r = base_rows;
        W.rows_i = 0;
        W.used = L.num_entries;
        W.over = false;
        W.fin = true;
        for (int k = lane; k < L.num_entries; k += 32) W.mr[L.entries[k].c * n + L.entries[k].r] = (uint16_t)k;
        for (int k = 0; k < L.num_entries; ++k) {
            const double v = L.values[(size_t)k * L.count + s];
            W.at(k) = v;
            W.check(v);
        }
        __syncwarp();
        const double wv = 2.0 * 3.141592653589793 * L.freqs[f];
        auto imag = [&](int r, int cc, double v, bool on) {
            if (r < 0 || cc < 0) return;
            const bool have = (__shfl_sync(0xffffffffu, W.rows_i, cc) >> r) & 1u;
            if (!have) W.at(W.add_slot(W.mi, W.rows_i, cc, r)) = 0.0;
            double& d = W.at(W.mi[cc * n + r]);
            if (on) d = d + v;
            W.check(d);
        };
        for (int k = 0; k < L.num_reacts; ++k) {
            const AcReact e = L.reacts[k];
            auto value = [&](int j) { return L.values[(size_t)(e.val + j) * L.count + s]; };
            auto cap = [&](int i, int j, double y, bool on) {
                imag(i, i, y, on), imag(j, j, y, on), imag(i, j, -y, on), imag(j, i, -y, on);
            };
            if (e.kind == SP_EL_C) {
                cap(e.n0, e.n1, wv * value(0), true);
            } else if (e.kind == SP_EL_L) {  // n0: its branch row
                imag(e.n0, e.n0, -(wv * value(0)), true);
            } else {
                const int pr[5][2] = {{e.n1, e.n2}, {e.n1, e.n0}, {e.n1, e.n3}, {e.n3, e.n2}, {e.n3, e.n0}};
                for (int q = 0; q < 5; ++q) {
                    const double gq = value(q);
                    cap(pr[q][0], pr[q][1], wv * gq, gq > 0.0);
                }
            }
        }
        for (int e = 0; e < c.num_elements; ++e) {
            const int kind = c.el[e].kind;
            if (kind == SP_EL_V && (L.source < 0 || L.source == e))
                W.acc(W.mr, W.rows_r, (__shfl_sync(0xffffffffu, W.rows_r, n) >> (nn + c.el[e].branch)) & 1u, n,
                      nn + c.el[e].branch, 1.0);
        }
        __syncwarp();

        // elimination, the right-hand side (column n) along with it
        bool ok = true;
        unsigned ones = 0;  // real pivots that are +-1 in every lane
        for (int i = 0; i < n; ++i) {
            const unsigned from = ~((1u << i) - 1u), below = ~((2u << i) - 1u);
            unsigned rr = __shfl_sync(0xffffffffu, W.rows_r, i), ri = __shfl_sync(0xffffffffu, W.rows_i, i);
            auto size = [&](int r) {
                const bool hr = (rr >> r) & 1u, hi = (ri >> r) & 1u;
                const double a = hr ? fabs(W.get(W.mr, i, r)) : 0.0, b = hi ? fabs(W.get(W.mi, i, r)) : 0.0;
                return (unsigned long long)__double_as_longlong(hr && hi ? a + b : hr ? a : b);
            };
            int piv = i;
            unsigned long long best = size(i);
            for (unsigned q = (rr | ri) & below; q; q &= q - 1) {
                const int r = __ffs(q) - 1;
                const unsigned long long v = size(r);
                if (v > best) best = v, piv = r;
            }
            const unsigned pset = __reduce_or_sync(0xffffffffu, 1u << piv), both = pset | (1u << i);
            if (pset != 1u << i && __popc(pset) == 1) {
                const int p = __ffs(pset) - 1;
                if (lane <= n) {  // lane c exchanges column c's two rows
                    uint16_t t = W.mr[lane * n + i];
                    W.mr[lane * n + i] = W.mr[lane * n + p], W.mr[lane * n + p] = t;
                    t = W.mi[lane * n + i];
                    W.mi[lane * n + i] = W.mi[lane * n + p], W.mi[lane * n + p] = t;
                    unsigned d = ((W.rows_r >> i) ^ (W.rows_r >> p)) & 1u;
                    W.rows_r ^= (d << i) | (d << p);
                    d = ((W.rows_i >> i) ^ (W.rows_i >> p)) & 1u;
                    W.rows_i ^= (d << i) | (d << p);
                }
                __syncwarp();
            } else if (pset != 1u << i) {
                // lanes pivot differently: every row involved gets a slot, each lane swaps its own two values
                for (int part = 0; part < 2; ++part) {
                    uint16_t* m = part ? W.mi : W.mr;
                    unsigned& rows = part ? W.rows_i : W.rows_r;
                    for (unsigned q = __ballot_sync(0xffffffffu, lane <= n && (rows & both)) & from; q; q &= q - 1) {
                        const int cc = __ffs(q) - 1;
                        const unsigned have = __shfl_sync(0xffffffffu, rows, cc);
                        for (unsigned z = both & ~have; z; z &= z - 1) W.at(W.add_slot(m, rows, cc, __ffs(z) - 1)) = 0.0;
                        double &a = W.at(m[cc * n + i]), &b = W.at(m[cc * n + piv]);
                        const double t = a;
                        a = b;
                        b = t;
                    }
                }
            }
            rr = __shfl_sync(0xffffffffu, W.rows_r, i), ri = __shfl_sync(0xffffffffu, W.rows_i, i);
            const bool dr_on = (rr >> i) & 1u, di_on = (ri >> i) & 1u;
            const double dre = dr_on ? W.get(W.mr, i, i) : 0.0, dim = di_on ? W.get(W.mi, i, i) : 0.0;
            ok = ok && best != 0;
            // 1 / diag = (dre - i dim) / ns
            double ire = dre, iim = 0.0;
            if (!di_on && __all_sync(0xffffffffu, dre == 1.0 || dre == -1.0)) {
                ones |= 1u << i;
            } else {
                const double ns = dr_on && di_on ? dre * dre + dim * dim : dr_on ? dre * dre : dim * dim;
                const double rn = best != 0 ? 1.0 / ns : 0.0;
                ire = dr_on && best != 0 ? warp_div(dre, ns, rn) : 0.0;
                iim = di_on && best != 0 ? warp_div(-dim, ns, rn) : 0.0;
                W.check(rn);
                int slot = W.used < W.cap ? W.used++ : W.cap - 1;
                if (slot == W.cap - 1) W.over = true;
                if (lane == 0) rns[i] = (uint16_t)slot;
                W.at(slot) = rn;
                __syncwarp();
            }
            const unsigned cols = __ballot_sync(0xffffffffu, lane <= n && (((W.rows_r | W.rows_i) >> i) & 1u)) & below;
            for (unsigned q = (rr | ri) & below; q; q &= q - 1) {
                const int r = __ffs(q) - 1;
                const bool ar_on = (rr >> r) & 1u, ai_on = (ri >> r) & 1u;
                const double ar = ar_on ? W.get(W.mr, i, r) : 0.0, ai = ai_on ? W.get(W.mi, i, r) : 0.0;
                // l = a / diag; a part is absent where its products are zero
                const bool rr1 = ar_on && dr_on, rr2 = ai_on && di_on, ii1 = ar_on && di_on, ii2 = ai_on && dr_on;
                const bool lr_on = rr1 || rr2, li_on = ii1 || ii2;
                const double lre = rr1 ? (rr2 ? ar * ire - ai * iim : ar * ire) : rr2 ? -(ai * iim) : 0.0;
                const double lim = ii1 ? (ii2 ? ar * iim + ai * ire : ar * iim) : ii2 ? ai * ire : 0.0;
                W.check(lre), W.check(lim);
                for (unsigned z = cols; z; z &= z - 1) {
                    const int cc = __ffs(z) - 1;
                    const unsigned cr = __shfl_sync(0xffffffffu, W.rows_r, cc), ci = __shfl_sync(0xffffffffu, W.rows_i, cc);
                    const bool ur_on = (cr >> i) & 1u, ui_on = (ci >> i) & 1u;
                    const double pr = ur_on ? -W.get(W.mr, cc, i) : 0.0, pi = ui_on ? -W.get(W.mi, cc, i) : 0.0;
                    const bool m1 = ur_on && lr_on, m2 = ui_on && li_on, m3 = ur_on && li_on, m4 = ui_on && lr_on;
                    if (m1 || m2)
                        W.acc(W.mr, W.rows_r, (cr >> r) & 1u, cc, r, m1 ? (m2 ? pr * lre - pi * lim : pr * lre) : -(pi * lim));
                    if (m3 || m4)
                        W.acc(W.mi, W.rows_i, (ci >> r) & 1u, cc, r, m3 ? (m4 ? pr * lim + pi * lre : pr * lim) : pi * lre);
                }
            }
        }
        // back substitution: unknown i replaces entry i of the right-hand side; its
        // parts' presence is the right-hand side's (column n) masks, extended
        unsigned xr_on = __shfl_sync(0xffffffffu, W.rows_r, n), xi_on = __shfl_sync(0xffffffffu, W.rows_i, n);
        for (int i = n - 1; i >= 0; --i) {
            const unsigned above = ~((2u << i) - 1u) & ((1u << n) - 1u);
            const unsigned colr = __ballot_sync(0xffffffffu, (W.rows_r >> i) & 1u) & above;
            const unsigned coli = __ballot_sync(0xffffffffu, (W.rows_i >> i) & 1u) & above;
            bool br_on = (xr_on >> i) & 1u, bi_on = (xi_on >> i) & 1u;
            double br = br_on ? W.get(W.mr, n, i) : 0.0, bi = bi_on ? W.get(W.mi, n, i) : 0.0;
            for (unsigned q = (colr | coli) & (xr_on | xi_on); q;) {
                const int cc = 31 - __clz(q);
                q ^= 1u << cc;
                const bool ar_on = (colr >> cc) & 1u, ai_on = (coli >> cc) & 1u, vr = (xr_on >> cc) & 1u, vi = (xi_on >> cc) & 1u;
                const double ar = ar_on ? W.get(W.mr, cc, i) : 0.0, ai = ai_on ? W.get(W.mi, cc, i) : 0.0;
                const double cr = vr ? -W.get(W.mr, n, cc) : 0.0, ci = vi ? -W.get(W.mi, n, cc) : 0.0;
                const bool m1 = vr && ar_on, m2 = vi && ai_on, m3 = vr && ai_on, m4 = vi && ar_on;
                if (m1 || m2) {
                    br = (m1 ? (m2 ? cr * ar - ci * ai : cr * ar) : -(ci * ai)) + br;
                    br_on = true;
                }
                if (m3 || m4) {
                    bi = (m3 ? (m4 ? cr * ai + ci * ar : cr * ai) : ci * ar) + bi;
                    bi_on = true;
                }
            }
            const bool dr_on = __shfl_sync(0xffffffffu, W.rows_r, i) >> i & 1u, di_on = __shfl_sync(0xffffffffu, W.rows_i, i) >> i & 1u;
            const double dr = dr_on ? W.get(W.mr, i, i) : 0.0, di = di_on ? W.get(W.mi, i, i) : 0.0;
            double qr, qi;
            bool qr_on = (br_on && dr_on) || (bi_on && di_on), qi_on = (bi_on && dr_on) || (br_on && di_on);
            if ((probed >> i) & 1u) {  // from all parts: a zero part gets the dense solve's sign
                const double ns = dr * dr + di * di;
                const double rn = (ones >> i) & 1u ? 1.0 : W.at(rns[i]);
                qr = warp_div(br * dr + bi * di, ns, rn);
                qi = warp_div(bi * dr - br * di, ns, rn);
                qr_on = qi_on = true;
            } else if ((ones >> i) & 1u) {
                qr = br * dr;
                qi = bi * dr;
            } else {
                const double ns = dr_on && di_on ? dr * dr + di * di : dr_on ? dr * dr : di * di, rn = W.at(rns[i]);
                const double nr = br_on && dr_on ? (bi_on && di_on ? br * dr + bi * di : br * dr) : bi_on && di_on ? bi * di : 0.0;
                const double ni = bi_on && dr_on ? (br_on && di_on ? bi * dr - br * di : bi * dr) : br_on && di_on ? -(br * di) : 0.0;
                qr = qr_on ? warp_div(nr, ns, rn) : 0.0;
                qi = qi_on ? warp_div(ni, ns, rn) : 0.0;
            }
            if (!ok) qr = qi = 0.0;
            W.check(qr), W.check(qi);
            if (qr_on) {
                if (!((xr_on >> i) & 1u)) W.add_slot(W.mr, W.rows_r, n, i);
                W.at(W.mr[n * n + i]) = qr;
                xr_on |= 1u << i;
            } else {
                xr_on &= ~(1u << i);
            }
            if (qi_on) {
                if (!((xi_on >> i) & 1u)) W.add_slot(W.mi, W.rows_i, n, i);
                W.at(W.mi[n * n + i]) = qi;
                xi_on |= 1u << i;
            } else {
                xi_on &= ~(1u << i);
            }
            __syncwarp();
        }
        if (live && (!W.fin || W.over)) {
            L.redo[s] = 1u;
            *L.any_redo = 1u;
        } else if (live) {
            if (!ok) atomicOr(L.singular + s, 1u);
            for (int k = 0; k < L.num_probe; ++k) {
                out[2 * k] = ok ? W.get(W.mr, n, L.probe[k]) : CUDART_NAN;
                out[2 * k + 1] = ok ? W.get(W.mi, n, L.probe[k]) : CUDART_NAN;
            }
        }
        __syncwarp();
    }
}
#endif  // SP_AC_KERNELS

}  // namespace sp
