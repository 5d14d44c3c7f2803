// What an AC system's elimination will need, from the circuit's pattern alone:
// the lists that the sparse kernel (ac_sparse.cuh) works on, and an estimate of
// its fill, by which the sweep picks its slots and its kernel.
#pragma once
#include <cstdint>
#include <utility>
#include <vector>

#include "ac.cuh"

namespace sp {

struct AcLists {
    std::vector<AcEntry> entries;  // real entries, ac_real_stamps' positions in order of first touch
    std::vector<AcReact> reacts;   // elements with imaginary ones
    int values = 0;                // their values
};

inline AcLists ac_lists(int n, int num_nodes, const sp_element* elements, int num_elements) {
    AcLists l;
    std::vector<char> seen((size_t)n * n, 0);
    auto put = [&](int r, int col) {
        if (r < 0 || col < 0 || seen[(size_t)col * n + r]) return;
        seen[(size_t)col * n + r] = 1;
        l.entries.push_back(AcEntry{(int16_t)r, (int16_t)col});
    };
    auto cond = [&](int i, int j) { put(i, i), put(j, j), put(i, j), put(j, i); };
    auto vccs = [&](int op, int on, int cp, int cn) { put(op, cp), put(op, cn), put(on, cp), put(on, cn); };
    for (int e = 0; e < num_elements; ++e) {
        const sp_element& el = elements[e];
        const int a0 = el.node[0], a1 = el.node[1], a2 = el.node[2], a3 = el.node[3], br = num_nodes + el.branch;
        switch (el.kind) {
            case SP_EL_R:
            case SP_EL_D: cond(a0, a1); break;
            case SP_EL_V:
            case SP_EL_L: put(a0, br), put(br, a0), put(a1, br), put(br, a1); break;
            case SP_EL_NMOS:
            case SP_EL_PMOS: cond(a0, a2), vccs(a0, a2, a1, a2); break;
            case SP_EL_NPN:
            case SP_EL_PNP: cond(a1, a2), cond(a0, a2), vccs(a0, a2, a1, a2); break;
            case SP_EL_BSIM3N:
            case SP_EL_BSIM3P: cond(a0, a2), vccs(a0, a2, a1, a2), vccs(a0, a2, a3, a2); break;
            default: break;
        }
        const bool b3 = el.kind == SP_EL_BSIM3N || el.kind == SP_EL_BSIM3P;
        if (el.kind != SP_EL_C && el.kind != SP_EL_L && !b3) continue;
        l.reacts.push_back(AcReact{el.kind, el.kind == SP_EL_L ? br : a0, a1, a2, a3, l.values});
        l.values += b3 ? 5 : 1;
    }
    for (AcReact& r : l.reacts) r.val += (int)l.entries.size();
    return l;
}

// Slots (parts of the matrix, its fill, the right-hand side and the unknowns,
// and the pivots' reciprocals) and FP64 operations of ac_sparse_kernel, and the
// dense kernel's operations, for an elimination on the pattern.  Pivots: an
// untouched +-1 of a source's or inductor's branch (larger than the conductances
// beside it), else the diagonal, else the first entry below.  Against numeric
// elimination with partial pivoting of 90 circuits of 5 to 28 unknowns: within 3
// slots and 4 % of the operations but for circuits of many transistors, whose
// pivots depend on the operating point (the op-amp: 83 slots estimated, 106).
struct AcFill {
    int slots = 0;
    long ops = 0, dense_ops = 0;
};

inline AcFill ac_fill(int n, int num_nodes, const sp_element* elements, int num_elements, const AcLists& l) {
    using Mask = uint32_t;  // the rows of a column
    std::vector<Mask> R(n + 1, 0), I(n + 1, 0), U(n + 1, 0);
    AcFill f;
    auto add = [&](Mask& m, int r) {
        f.slots += !(m >> r & 1);
        m |= Mask(1) << r;
    };
    for (const AcEntry& e : l.entries) add(R[e.c], e.r);
    auto imag = [&](int r, int c) {
        if (r >= 0 && c >= 0) add(I[c], r);
    };
    auto cap = [&](int i, int j) { imag(i, i), imag(j, j), imag(i, j), imag(j, i); };
    for (const AcReact& e : l.reacts) {
        if (e.kind == SP_EL_C) cap(e.n0, e.n1);
        else if (e.kind == SP_EL_L) imag(e.n0, e.n0);
        else cap(e.n1, e.n2), cap(e.n1, e.n0), cap(e.n1, e.n3), cap(e.n3, e.n2), cap(e.n3, e.n0);
    }
    for (int e = 0; e < num_elements; ++e) {
        const sp_element& el = elements[e];
        if (el.kind != SP_EL_V && el.kind != SP_EL_L) continue;
        const int br = num_nodes + el.branch;
        for (int k = 0; k < 2; ++k)
            if (el.node[k] >= 0) U[br] |= Mask(1) << el.node[k], U[el.node[k]] |= Mask(1) << br;
        if (el.kind == SP_EL_V) add(R[n], br);
    }
    auto first = [](Mask m) { return __builtin_ctz(m); };
    for (int i = 0; i < n; ++i) {
        const Mask from = ~((Mask(1) << i) - 1), unit = U[i] & from, any = (R[i] | I[i]) & from;
        const int p = unit ? (unit >> i & 1 ? i : first(unit)) : any ? first(any) : i;
        if (p != i)
            for (std::vector<Mask>* m : {&R, &I, &U})
                for (Mask& c : *m) {
                    const Mask d = (c >> i ^ c >> p) & 1;
                    c ^= d << i | d << p;
                }
        const bool one = U[i] >> i & 1 && !(I[i] >> i & 1);
        f.slots += !one;
        f.ops += one ? 10 : 30;  // a unit pivot divides nothing
        f.dense_ops += 30 + 6L * (n - 1 - i) + 8L * (n - 1 - i) * (n - i);
        const bool dr = R[i] >> i & 1, di = I[i] >> i & 1;
        for (Mask q = (R[i] | I[i]) & (from << 1); q; q &= q - 1) {
            const int r = first(q);
            const bool ar = R[i] >> r & 1, ai = I[i] >> r & 1;
            const int lr = (ar && dr) + (ai && di), li = (ar && di) + (ai && dr);
            f.ops += lr + li + (lr == 2) + (li == 2);
            for (int c = i + 1; c <= n; ++c) {
                const bool ur = R[c] >> i & 1, ui = I[c] >> i & 1;
                const int re = (ur && lr) + (ui && li), im = (ur && li) + (ui && lr);
                f.ops += re + im + (re == 2) + (im == 2) + (re > 0) + (im > 0);
                if (re) add(R[c], r);
                if (im) add(I[c], r);
                if (re || im) U[c] &= ~(Mask(1) << r);
            }
        }
    }
    Mask xr = R[n], xi = I[n];  // the unknowns' parts, in the right-hand side's slots
    for (int i = n - 1; i >= 0; --i) {
        bool br = xr >> i & 1, bi = xi >> i & 1;
        for (int c = i + 1; c < n; ++c) {
            const bool ar = R[c] >> i & 1, ai = I[c] >> i & 1, vr = xr >> c & 1, vi = xi >> c & 1;
            br = br || (vr && ar) || (vi && ai);
            bi = bi || (vr && ai) || (vi && ar);
        }
        const bool dr = R[i] >> i & 1, di = I[i] >> i & 1;
        const bool qr = (br && dr) || (bi && di), qi = (bi && dr) || (br && di);
        f.slots += (qr && !(xr >> i & 1)) + (qi && !(xi >> i & 1));
        xr = (xr & ~(Mask(1) << i)) | Mask(qr) << i;
        xi = (xi & ~(Mask(1) << i)) | Mask(qi) << i;
    }
    return f;
}

}  // namespace sp
