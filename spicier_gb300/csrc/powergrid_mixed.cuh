// Power-grid corner sweep, SP_PREC_MIXED: the FP32 Krylov solves with the
// whole basis on chip.
//
// The arithmetic is that of powergrid.cuh's GMRES, element by element and sum
// by sum (results and step counts are the same as those of a kernel of that
// form in FP32): rows p = t (mod 512) are summed in order, 32 such sums (t =
// 32 w ... 32 w + 31, "row group" w) by an exchange tree and the 16 groups'
// sums in order (the norm's by the same tree again).  A thread owns the rows
// of t and t + 256, so that every step of its sums is one packed FP32 pair.
//
// What bounds it: the number of Arnoldi steps (8,200 per corner on the 64 x 64
// mesh, each reading k + 1 basis vectors four times) and what a step cannot
// overlap.  With the basis in L2 a step took 148,000 cycles, 120,000 of them
// waiting for basis vectors, 9,000 in the Givens rotations of one thread and
// 5,000 in an FP64 square root and division done by every thread.  Here it
// takes 18,000 (six in projections, five in subtractions, three in the
// stencil), and each restart 165,000 more, most of it FP64 chains:
//  * a thread's elements of the first vectors are its private words of tensor
//    memory (256 KB: 16 vectors of 16 rows a thread, or all of them on meshes
//    of up to 2,048 unknowns), those of the next ones (ten beside the edges of
//    a 64 x 64 mesh) its words of shared memory, and only what is left is in
//    global memory.  Rows 4,096 and up (at least one on a 64 x 64 mesh) lie in
//    shared memory, so that the other threads do no work for them;
//  * the sums of eight projections share an exchange tree (nine shuffles
//    instead of forty, each sum with the same terms in the same order), and
//    every warp adds the groups' sums for itself, so a pass has one barrier;
//  * the warp beyond the rows does the FP64 part of step k (Hessenberg column,
//    Givens rotations, convergence test) while the others do step k + 1, which
//    is thrown away where step k turns out to be the last;
//  * 1 / sqrt comes from FP32 pairs, FP64 only where that could round
//    differently.
// Eight warps of rows and one more: with sixteen and one, a quarter of the SM
// holds five warps and the registers end at 96, which spilled basis vectors
// (270 against 214 ms; 27,000 cycles a step).
// 256 corners of the 64 x 64 mesh: 1,430 ms before, 214 now.
#pragma once
#include "fpconv.cuh"
#include "newton_dense.cuh"
#include "powergrid.cuh"
#include <type_traits>

namespace sp {

constexpr int kGridRowThreads = kGridThreads / 2;
constexpr int kGridMixedThreads = kGridRowThreads + 32;  // and the warp of the FP64 column
constexpr int kGridGroups = kGridThreads / 32;           // row groups: warp w has w and w + 8
constexpr int kGridProjLd = kGridMaxRestart + 1;

// Pairs of rows per thread in registers: the smallest of 2, 4, 8 that covers
// the mesh (at 8, rows past 4,096 are the tail).
__host__ __device__ inline int grid_mixed_rows(int n) {
    return n <= 2 * kGridThreads ? 2 : (n <= 4 * kGridThreads ? 4 : 8);
}

// Byte offsets in dynamic shared memory: what does not depend on the mesh ...
constexpr int kGridHmat = 0;
constexpr int kGridGvec = kGridHmat + 8 * kGridMaxRestart * kGridProjLd;
constexpr int kGridCs = kGridGvec + 8 * (kGridMaxRestart + 1);
constexpr int kGridSn = kGridCs + 8 * kGridMaxRestart;
constexpr int kGridYv = kGridSn + 8 * kGridMaxRestart;
constexpr int kGridRcp = kGridYv + 8 * kGridMaxRestart;
constexpr int kGridRedd = kGridRcp + 8 * kGridMaxRestart;
constexpr int kGridKept = kGridRedd + 8 * 32;
constexpr int kGridHcol = kGridKept + 8 * 4;
constexpr int kGridRed = kGridHcol + 4 * 4 * kGridMaxRestart;
constexpr int kGridProj = kGridRed + 4 * 64;
constexpr int kGridNorm = kGridProj + 4 * 2 * kGridGroups * kGridProjLd;
constexpr int kGridFlags = kGridNorm + 4 * 2 * 32;
constexpr int kGridZs = (kGridFlags + 16 + 15) & ~15;

// ... and what does; slots: basis vectors kept there.
struct GridMixedSmem {
    int tail;  // rows past 8 * 512
    int slots;
    size_t edges, tails, basis, total;
};

__host__ __device__ inline GridMixedSmem grid_mixed_smem(int n, int m, int max_smem) {
    const int nq = grid_mixed_rows(n);
    GridMixedSmem s;
    s.tail = n > 8 * kGridThreads ? n - 8 * kGridThreads : 0;
    size_t o = kGridZs + 4 * ((size_t)nq * kGridThreads + s.tail);
    s.edges = o; o += 4 * 2 * ((size_t)nq * kGridThreads + s.tail);
    s.tails = o; o += 4 * (size_t)((m + 7) & ~7) * s.tail;
    s.basis = o = (o + 15) & ~size_t(15);
    s.slots = 0;
    if (nq == 8 && m > 16) {  // the vectors that tensor memory does not hold, in pairs
        const size_t vec = 4 * 8 * kGridThreads;
        const int need = (m - 16 + 1) & ~1;
        const int fit = (size_t)max_smem > o ? (int)(((size_t)max_smem - o) / vec) & ~1 : 0;
        s.slots = need < fit ? need : fit;
        o += vec * s.slots;
    }
    s.total = o;
    return s;
}

#ifdef SP_KERNEL_NS
namespace SP_KERNEL_NS {

// Tensor memory as private words: a warp reaches lanes 32 (warp % 4) ..., one
// 32-bit word per thread and column.
template <int N>
__device__ __forceinline__ void tmem_read(uint32_t addr, float* v);
template <int N>
__device__ __forceinline__ void tmem_write(uint32_t addr, const float (&v)[N]);

template <>
__device__ __forceinline__ void tmem_read<8>(uint32_t addr, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
          "=f"(v[6]), "=f"(v[7])
        : "r"(addr)
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_read<16>(uint32_t addr, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
          "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),
          "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(addr)
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_read<32>(uint32_t addr, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]),
          "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),
          "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]),
          "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
          "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]),
          "=f"(v[30]), "=f"(v[31])
        : "r"(addr)
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_write<4>(uint32_t addr, const float (&v)[4]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n\ttcgen05.wait::st.sync.aligned;" ::"r"(addr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3])
        : "memory");
}
template <>
__device__ __forceinline__ void tmem_write<8>(uint32_t addr, const float (&v)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(addr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
        : "memory");
}

template <>
__device__ __forceinline__ void tmem_write<16>(uint32_t addr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(addr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
        : "memory");
}

// c + a * b, two at a time
__device__ __forceinline__ void fma_pair(float& c0, float& c1, float a0, float a1, float b0, float b1) {
    uint64_t a, b, c;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(a0), "f"(a1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
    asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(c0), "f"(c1));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(c0), "=f"(c1) : "l"(c));
}

// The threads that own rows.
__device__ __forceinline__ void grid_rows_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// The sum of 512 partial sums, (a, b) from threads t and t + 256 of the row
// numbering: block_sum of a 512-thread block.
__device__ inline float grid_block_sum(float a, float b, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();  // red[] free
    if (lane == 0 && warp < kGridGroups / 2) {
        red[warp] = a;
        red[warp + kGridGroups / 2] = b;
    }
    __syncthreads();
    float s = lane < kGridGroups ? red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// (float)(1 / sqrt((double)s)): y0 (within 2^-22) plus its correction from the
// exact remainder, good to 2^-42; FP64 where that leaves the rounding in doubt
// (or s is far from 1).
__device__ __noinline__ static float grid_inv_sqrt_fp64(float s) { return (float)(1.0 / sqrt((double)s)); }
__device__ __forceinline__ float grid_inv_sqrt(float s) {
    const float y0 = rsqrtf(s), h = s * y0, l = fmaf(s, y0, -h);
    const float t = fmaf(-l, y0, fmaf(-h, y0, 1.0f));  // 1 - s y0^2
    const float d = y0 * t * fmaf(0.375f, t, 0.5f);
    const float y = y0 + d, e = (y0 - y) + d;
    const unsigned yb = __float_as_uint(y);
    const float ulp = __uint_as_float((yb & 0x7f800000u) - (23u << 23));
    const bool sure = s >= 0x1p-90f && s <= 0x1p90f && (yb & 0x7fffffu) && fabsf(fabsf(e) - 0.5f * ulp) > 0x1p-14f * ulp;
    return sure ? y : grid_inv_sqrt_fp64(s);
}

// Exact for the numbers that grid_widens takes, zero and the normal ones (FP64
// conversions would queue for the FP64 pipe).
__device__ __forceinline__ bool grid_widens(float x) {
    const unsigned mag = __float_as_uint(x) & 0x7fffffffu;
    return mag - 0x00800000u < 0x7f000000u || mag == 0;
}
__device__ __forceinline__ double grid_widen(float x) {
    const unsigned f = __float_as_uint(x), mag = f & 0x7fffffffu;
    return __hiloint2double((int)((f & 0x80000000u) | (mag ? (mag >> 3) + 0x38000000u : 0u)), (int)(mag << 29));
}

// The instance, read anew: what a solve needs once per restart is worked out
// again from it there (kept in registers it would be spilled around the
// Arnoldi steps, and 28 KB of L1 beside 227 KB of shared memory do not hold
// the stacks).
__device__ __forceinline__ uint32_t grid_instance() {
    uint32_t i;
    asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(i));
    return i;
}
__device__ __forceinline__ GridPtrs grid_instance_ptrs(const GridLaunch& L) {
    return grid_ptrs(L, grid_ws(L.cfg, 4), grid_instance());
}

template <int NQ>
struct GridBasis {
    static constexpr int kRows = 2 * NQ;             // rows t + 256 r, r < kRows
    static constexpr int kTmem = NQ == 8 ? 16 : 32;  // vectors in tensor memory
    uint32_t tmem;                                   // this thread's words
    float4* sm;                                      // this thread's words: [slot][kRows / 4][256]
    int slots;
    float* glob;  // [vector][n]
    int n, tid;

    // Vectors j0 and j0 + 1 (j0 even; past k: anything): v[u * kRows + r] is
    // row r of vector j0 + u.  SRC: all in tensor memory (0), in shared memory
    // (1) or in global memory (2); each source has its own copy of the loops.
    template <int SRC>
    __device__ __forceinline__ void load2(int j0, int k, float (&v)[2 * kRows]) const {
        if (SRC == 0) {
            __syncwarp();  // aligned: all lanes together
            tmem_read<2 * kRows>(tmem + (uint32_t)(j0 * kRows), v);
        } else if (SRC == 1) {
#pragma unroll
            for (int u = 0; u < kRows / 2; ++u) {
                const float4 x = sm[(size_t)((j0 - kTmem) * (kRows / 4) + u) * kGridRowThreads];
                v[4 * u] = x.x;
                v[4 * u + 1] = x.y;
                v[4 * u + 2] = x.z;
                v[4 * u + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    const int p = tid + r * kGridRowThreads;
                    v[u * kRows + r] = j0 + u <= k && p < n ? glob[(size_t)(j0 + u) * n + p] : 0.f;
                }
        }
    }
    // f(source, count, j0) for the vectors 0 .. k, count (at most M) at a time
    template <int M, class F>
    __device__ __forceinline__ void each(int k, F&& f) const {
        using std::integral_constant;
        int j0 = 0;
        for (; j0 <= k && j0 < kTmem; j0 += M) f(integral_constant<int, 0>(), integral_constant<int, M>(), j0);
        if (NQ == 8) {
            for (; j0 <= k && j0 + M <= kTmem + slots; j0 += M)
                f(integral_constant<int, 1>(), integral_constant<int, M>(), j0);
            if (M > 2)
                for (; j0 <= k && j0 < kTmem + slots; j0 += 2)
                    f(integral_constant<int, 1>(), integral_constant<int, 2>(), j0);
            for (; j0 <= k; j0 += 2) f(integral_constant<int, 2>(), integral_constant<int, 2>(), j0);
        }
    }
    __device__ __forceinline__ void store(int j, const float (&v)[kRows]) const {
        if (NQ < 8 || j < kTmem) {
            __syncwarp();
            tmem_write<kRows>(tmem + (uint32_t)(j * kRows), v);
        } else if (j - kTmem < slots) {
#pragma unroll
            for (int u = 0; u < kRows / 4; ++u)
                sm[(size_t)((j - kTmem) * (kRows / 4) + u) * kGridRowThreads] =
                    make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
        } else {
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int p = tid + r * kGridRowThreads;
                if (p < n) glob[(size_t)j * n + p] = v[r];
            }
        }
    }
};

template <int NQ>
__global__ void __launch_bounds__(kGridMixedThreads, 1) grid_mixed_kernel(GridLaunch L) {
    extern __shared__ __align__(16) unsigned char gsm[];
    const sp_grid_config& c = L.cfg;
    const int Cn = c.cols, R = c.rows, n = R * Cn + 1, nn = n - 1, m = c.restart;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int T = kGridRowThreads, NR = 2 * NQ;
    const bool rows = tid < T;  // the last warp owns none
    const int p0 = grid_first<T>(n);
    auto inst = [&]() { return (uint32_t)(L.first + grid_instance()); };
    auto iterate = [&]() { return L.x + (size_t)grid_instance() * n; };
    const GridMixedSmem S = grid_mixed_smem(n, m, L.max_smem);
    double* hmat = (double*)(gsm + kGridHmat);
    double* gvec = (double*)(gsm + kGridGvec);
    double* cs = (double*)(gsm + kGridCs);
    double* sn = (double*)(gsm + kGridSn);
    double* yv = (double*)(gsm + kGridYv);
    double* rcp = (double*)(gsm + kGridRcp);  // 1 / diagonal of the rotated columns
    double* redd = (double*)(gsm + kGridRedd);
    float* hcol = (float*)(gsm + kGridHcol);  // [step parity][pass][kGridMaxRestart]
    float* red = (float*)(gsm + kGridRed);
    float* proj = (float*)(gsm + kGridProj);  // [pass][warp][kGridProjLd]
    float* norm = (float*)(gsm + kGridNorm);  // [step parity][32]
    int* done = (int*)(gsm + kGridFlags);     // [step parity]
    uint32_t* tmem_slot = (uint32_t*)(gsm + kGridFlags) + 2;
    float* zs = (float*)(gsm + kGridZs);
    // the tail rows, T apart
    const bool tail[2] = {tid < S.tail && rows, tid + T < S.tail && rows}, warp_tail = warp * 32 < S.tail && rows;
    float* tails = (float*)(gsm + S.tails);  // [vector][S.tail]
    const int tt[2] = {tail[0] ? tid : 0, tail[1] ? tid + T : 0}, pt = NR * T + tid;
    double* kept = (double*)(gsm + kGridKept);                  // ||b||, tolerance, KCL residual

    constexpr uint32_t kColumns = 2 * NR * GridBasis<NQ>::kTmem;  // 512, or 256
    if (warp == T / 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(tmem_slot)),
                     "r"(kColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_draws<T>(L, grid_instance_ptrs(L), inst(), iterate());
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    GridBasis<NQ> V;
    V.tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * NR * GridBasis<NQ>::kTmem);
    V.sm = (float4*)(gsm + S.basis) + tid;
    V.slots = S.slots;
    V.glob = (float*)grid_instance_ptrs(L).V;
    V.n = n;
    V.tid = tid;
    // FP32 edge conductances: gh[p] from p to p + 1, gv[p] from p to the row below
    float* gh = (float*)(gsm + S.edges);
    const int padded = NR * T + S.tail;  // both padded like z, so that no row's loads need a test
    float* gv = gh + padded;
    {
        const GridPtrs g = grid_instance_ptrs(L);
        for (int p = grid_first<T>(padded); p < padded; p += T) {
            const int rr = p / Cn;
            gh[p] = p < nn && p - rr * Cn < Cn - 1 ? (float)g.gh[p - rr] : 0.f;
            gv[p] = p < nn && rr < R - 1 ? (float)g.gv[p] : 0.f;
        }
    }
    const float strap = (float)c.strap_g;
    const int c1 = Cn - 1, c2 = (R - 1) * Cn, c3 = nn - 1;
    uint64_t edges = 0;    // 4 bits a row: left, right, up, down
    unsigned special = 0;  // 1 bit a row: strap nodes and the branch row
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int p = tid + r * T;
        if (!rows || p >= n) continue;
        const int rr = p / Cn, j = p - rr * Cn;
        if (p < nn)
            edges |= (uint64_t)((unsigned)(j > 0) | (unsigned)(j < Cn - 1) << 1 | (unsigned)(rr > 0) << 2 |
                                (unsigned)(rr < R - 1) << 3)
                     << (4 * r);
        if (p == nn || p == 0 || p == c1 || p == c2 || p == c3) special |= 1u << r;
    }
    auto edge = [&](int r) { return (unsigned)(edges >> (4 * r)); };

    int newton_it = 0, krylov_total = 0;
    uint8_t status = SP_ST_FAILED;
    auto vto = [&]() { return grid_vto(c, inst()); };
    auto beta = [&]() { return c.kp * 1.0 * c.w / c.l; };  // level1.rs:68-70 (NF = 1)
    for (int it = 1; it <= c.max_newton; ++it) {
        grid_linearise<T>(c, grid_instance_ptrs(L), vto(), beta(), iterate());
        float inv[NR], dT[NR], inv_t[2] = {0.f, 0.f}, dT_t[2] = {0.f, 0.f};
        {
            const GridPtrs g = grid_instance_ptrs(L);
            const double* x = iterate();
            auto jacobi = [&](int p, float& iv, float& d) {
                const double dg = g.diag[p];
                iv = (float)(fabs(dg) < 1e-30 ? 1.0 : 1.0 / dg);
                d = (float)dg;
            };
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const int p = tid + r * T;
                inv[r] = dT[r] = 0.f;
                if (rows && p < n) jacobi(p, inv[r], dT[r]);
                asm volatile("" ::: "memory");
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (tail[h]) jacobi(pt + h * T, inv_t[h], dT_t[h]);
            // --- right-hand side b - A x, in FP64
            double rmax = 0.0;
            float bb[2] = {0.f, 0.f};
            bool odd = false;
            for (int p = p0; p < n; p += T, odd = !odd) {
                const double rv = g.b[p] - grid_apply_row<double>(c, g.gh, g.gv, g.diag, x, p);
                g.r[p] = rv;
                if (p < nn) rmax = fmax(rmax, fabs(rv));
                const float rf = (float)rv;
                if (odd) bb[1] += rf * rf;
                else bb[0] += rf * rf;
            }
            // --- GMRES on A d = r; d is accumulated in b's storage (b is no longer needed)
            for (int p = p0; p < n; p += T) g.b[p] = 0.0;
            rmax = block_max<T>(rmax, redd);
            const double b_norm = sqrt((double)grid_block_sum(bb[0], bb[1], red));
            if (tid == 0) {
                kept[0] = b_norm;
                // FP32 Krylov: each solve only has to gain three digits; the FP64
                // residual of the next Newton iteration refines the rest
                kept[1] = fmax(c.krylov_tol, 1e-3);
                kept[2] = rmax;  // the KCL residual of the current iterate
            }
            __syncthreads();
        }
        int total = 0;
        bool solved = kept[0] < 1e-30;
        for (int cycle = 0; !solved && cycle < c.max_krylov; ++cycle) {
            // residual of the current solution, r - A sol, in FP64 (an FP32
            // difference of two nearly equal vectors would stall the restarts)
            __syncthreads();
            float v[NR], v_t[2] = {0.f, 0.f}, loc[2] = {0.f, 0.f};
            const GridPtrs g = grid_instance_ptrs(L);
            const double* sol = g.b;
            // grid_apply_row without branches around its loads (a neighbour that is
            // not there: the row itself)
            auto apply64 = [&](int p, unsigned e4) {
                const int rr = p / Cn, pl = e4 & 1 ? p - 1 : p, pr = e4 & 2 ? p + 1 : p;
                const int pu = e4 & 4 ? p - Cn : p, pd = e4 & 8 ? p + Cn : p;
                const double d = g.diag[p], xp = sol[p], xl = sol[pl], xr = sol[pr], xu = sol[pu], xd = sol[pd];
                const double hl = g.gh[e4 & 1 ? p - rr - 1 : 0], hr = g.gh[e4 & 2 ? p - rr : 0];
                const double vu = g.gv[e4 & 4 ? pu : 0], vd = g.gv[e4 & 8 ? p : 0];
                double t = d * xp;
                t = e4 & 1 ? fma(-hl, xl, t) : t;
                t = e4 & 2 ? fma(-hr, xr, t) : t;
                t = e4 & 4 ? fma(-vu, xu, t) : t;
                t = e4 & 8 ? fma(-vd, xd, t) : t;
                return t;
            };
            if (rows) {
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int p = tid + r * T;
                    const int pv = p < n ? p : n - 1;
                    const float t = (float)(g.r[pv] - apply64(pv, p < n ? edge(r) : 0u));
                    v[r] = p < n ? t : 0.f;
                    if (r & 1) asm volatile("" ::: "memory");  // two rows' loads at a time: registers
                }
                if (special) {
#pragma unroll
                    for (int r = 0; r < NR; ++r)
                        if (special >> r & 1) {
                            const int p = tid + r * T;
                            v[r] = (float)(g.r[p] - grid_apply_row<double>(c, g.gh, g.gv, g.diag, sol, p));
                        }
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) loc[r & 1] += v[r] * v[r];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (tail[h]) {
                        const int p = pt + h * T;
                        v_t[h] = (float)(g.r[p] - grid_apply_row<double>(c, g.gh, g.gv, g.diag, sol, p));
                        loc[h] += v_t[h] * v_t[h];
                    }
            }
            const double r_norm = sqrt((double)grid_block_sum(loc[0], loc[1], red));
            if (r_norm / kept[0] < kept[1]) {
                solved = true;
                break;
            }
            const float inv_r = (float)(1.0 / r_norm);
            if (rows) {
#pragma unroll
                for (int r = 0; r < NR; ++r) v[r] *= inv_r;
                V.store(0, v);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    v_t[h] *= inv_r;
                    if (tail[h]) tails[tt[h]] = v_t[h];
                }
            } else {
                gvec[lane] = lane == 0 ? r_norm : 0.0;
                if (lane == 0) gvec[32] = 0.0;
                __syncwarp();
            }

            // the FP64 part of step k, by the last warp: Hessenberg column,
            // rotations (lane j has row j; only the value carried from row to
            // row is a chain), convergence test
            auto column = [&](int k) {
                const float* hc = hcol + (k & 1) * 2 * kGridMaxRestart;
                double* hk = hmat + k * kGridProjLd;
                const double h = (double)hc[lane] + (double)hc[kGridMaxRestart + lane];  // lanes past k: unused
                float s = lane < kGridGroups ? norm[(k & 1) * 32 + lane] : 0.f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                const double w_norm = sqrt((double)s);
                if (s == 0.f) {  // breakdown: the column stays as it is
                    if (lane <= k) hk[lane] = h;
                    if (lane == k) rcp[k] = 1.0 / h;
                    __syncwarp();
                    return;
                }
                const double hn = __shfl_down_sync(0xffffffffu, h, 1);
                const double cj = lane < k ? cs[lane] : 0.0, sj = lane < k ? sn[lane] : 0.0;
                // the products are rounded or fused as in the one-thread form of
                // the rotation (the test for the last step hangs on their bits)
                double carry = __shfl_sync(0xffffffffu, h, 0), mine = carry;
                for (int j = 0; j < k; ++j) {
                    const double sjj = __shfl_sync(0xffffffffu, sj, j), cjj = __shfl_sync(0xffffffffu, cj, j);
                    const double hj1 = __shfl_sync(0xffffffffu, hn, j);
                    carry = __fma_rn(cjj, hj1, -__dmul_rn(sjj, carry));
                    if (lane == j + 1) mine = carry;
                }
                const double rot = __fma_rn(cj, mine, __dmul_rn(sj, hn));
                const double hkk = carry, hk1 = w_norm;
                double cc = 1.0, ss = 0.0;
                if (fabs(hk1) >= 1e-30) {
                    const double rr2 = sqrt(__fma_rn(hkk, hkk, __dmul_rn(hk1, hk1)));
                    const double quo = (lane & 1 ? hk1 : hkk) / rr2;
                    cc = __shfl_sync(0xffffffffu, quo, 0);
                    ss = __shfl_sync(0xffffffffu, quo, 1);
                }
                const double hd = __fma_rn(cc, hkk, __dmul_rn(ss, hk1));
                const double g0 = gvec[k], g1 = gvec[k + 1];
                const double gk1 = -ss * g0 + cc * g1, gk = cc * g0 + ss * g1;  // g1 is 0
                const double quo = (lane & 1 ? 1.0 : fabs(gk1)) / (lane & 1 ? hd : kept[0]);
                __syncwarp();
                if (lane < k) hk[lane] = rot;
                if (lane == 0) {
                    cs[k] = cc;
                    sn[k] = ss;
                    hk[k] = hd;
                    gvec[k] = gk;
                    gvec[k + 1] = gk1;
                    done[k & 1] = quo < kept[1];
                }
                if (lane == 1) rcp[k] = quo;
                __syncwarp();
            };

            int k = 0;
            for (;;) {
                // steps 0 .. k - 1 are counted, and the last of them still
                // has its column to come
                if (k == m || total + 1 > c.max_krylov) {
                    if (k > 0) {
                        if (!rows) column(k - 1);
                        __syncthreads();
                        if (!done[(k - 1) & 1] && k < m) ++total;
                    } else {
                        ++total;
                    }
                    break;
                }
                float w[NR], w_t[2] = {0.f, 0.f};
                if (rows) {
                    // z_k = M^-1 v_k into shared memory; w = A z_k
#pragma unroll
                    for (int r = 0; r < NR; ++r) zs[tid + r * T] = v[r] = v[r] * inv[r];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (tail[h]) zs[pt + h * T] = v_t[h] * inv_t[h];
                    grid_rows_sync();
                    // (a neighbour that is not there is read all the same: what lies
                    // before z and after the edges is shared memory of this block)
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const int p = tid + r * T;
                        const unsigned e4 = edge(r);
                        const float zl = zs[p - 1], zr = zs[p + 1], zu = zs[p - Cn], zd = zs[p + Cn];
                        const float el = gh[p - 1], er = gh[p], eu = gv[p - Cn], ed = gv[p];
                        float t = dT[r] * v[r];
                        t = e4 & 1 ? fmaf(-el, zl, t) : t;
                        t = e4 & 2 ? fmaf(-er, zr, t) : t;
                        t = e4 & 4 ? fmaf(-eu, zu, t) : t;
                        t = e4 & 8 ? fmaf(-ed, zd, t) : t;
                        w[r] = t;
                    }
                    auto straps = [&](int p, float t) {
                        if (p == nn) {
                            t = zs[0];
                        } else if (p == 0) {
                            t -= strap * zs[c1];
                            t -= strap * zs[c2];
                            t -= strap * zs[c3];
                            t += zs[nn];
                        } else if (p == c1 || p == c2 || p == c3) {
                            t -= strap * zs[0];
                        }
                        return t;
                    };
                    if (special) {
#pragma unroll
                        for (int r = 0; r < NR; ++r)
                            if (special >> r & 1) w[r] = straps(tid + r * T, w[r]);
                    }
                    if (NQ == 8 && warp_tail) {
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (tail[h]) {
                                const int p = pt + h * T, rr = p / Cn, j = p - rr * Cn;
                                if (p < nn) {
                                    w_t[h] = dT_t[h] * zs[p];
                                    if (j > 0) w_t[h] -= gh[p - 1] * zs[p - 1];
                                    if (j < Cn - 1) w_t[h] -= gh[p] * zs[p + 1];
                                    if (rr > 0) w_t[h] -= gv[p - Cn] * zs[p - Cn];
                                    if (rr < R - 1) w_t[h] -= gv[p] * zs[p + Cn];
                                }
                                w_t[h] = straps(p, w_t[h]);
                            }
                    }
                    // classical Gram-Schmidt, applied twice (CGS2): one block
                    // reduction of all k+1 projections per pass instead of one per
                    // basis vector; in exact arithmetic the same Hessenberg column
                    // as modified Gram-Schmidt, and as well conditioned in practice
                    for (int pass = 0; pass < 2; ++pass) {
                        float* pr = proj + pass * kGridGroups * kGridProjLd;
                        V.template each<8>(k, [&](auto src, auto count, int j0) {
                            // (vectors past k: anything, for sums that are dropped)
                            constexpr int G = decltype(count)::value;
                            float acc[G], acc2[G];  // of the two row groups
#pragma unroll
                            for (int u = 0; u < G; ++u) acc[u] = acc2[u] = 0.f;
#pragma unroll
                            for (int part = 0; part < G; part += 2) {
                                float e[2 * NR];
                                V.template load2<decltype(src)::value>(j0 + part, k, e);
#pragma unroll
                                for (int r = 0; r < NR; r += 2)
#pragma unroll
                                    for (int u = 0; u < 2; ++u)
                                        fma_pair(acc[part + u], acc2[part + u], e[u * NR + r], e[u * NR + r + 1], w[r],
                                                 w[r + 1]);
                            }
                            if (NQ == 8 && warp_tail) {
#pragma unroll
                                for (int u = 0; u < G; ++u) {
                                    const float et = tails[(j0 + u) * S.tail + tt[0]];
                                    acc[u] += (tail[0] ? et : 0.f) * w_t[0];
                                }
                                if (S.tail > T) {
#pragma unroll
                                    for (int u = 0; u < G; ++u) {
                                        const float et = tails[(j0 + u) * S.tail + tt[1]];
                                        acc2[u] += (tail[1] ? et : 0.f) * w_t[1];
                                    }
                                }
                            }
                            // sums over the row groups: each exchange halves the vectors a
                            // lane adds up, lanes 32 / G * u ... end with vector j0 + u's
                            int o = 16;
#pragma unroll
                            for (int left = G / 2; left > 0; left /= 2, o /= 2) {
                                const bool high = lane & o;
#pragma unroll
                                for (int u = 0; u < left; ++u) {
                                    const float give = high ? acc[u] : acc[u + left];
                                    acc[u] = (high ? acc[u + left] : acc[u]) + __shfl_xor_sync(0xffffffffu, give, o);
                                    const float give2 = high ? acc2[u] : acc2[u + left];
                                    acc2[u] = (high ? acc2[u + left] : acc2[u]) + __shfl_xor_sync(0xffffffffu, give2, o);
                                }
                            }
#pragma unroll
                            for (; o > 0; o /= 2) {
                                acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
                                acc2[0] += __shfl_xor_sync(0xffffffffu, acc2[0], o);
                            }
                            const int ju = j0 + lane / (32 / G);
                            if (lane % (32 / G) == 0 && ju <= k) {
                                pr[warp * kGridProjLd + ju] = acc[0];
                                pr[(warp + kGridGroups / 2) * kGridProjLd + ju] = acc2[0];
                            }
                        });
                        grid_rows_sync();
                        float hs = 0.f;
                        if (lane <= k)
#pragma unroll
                            for (int w2 = 0; w2 < kGridGroups; ++w2) hs += pr[w2 * kGridProjLd + lane];
                        if (warp == 0) hcol[((k & 1) * 2 + pass) * kGridMaxRestart + lane] = hs;
                        V.template each<2>(k, [&](auto src, auto, int j0) {
                            float e[2 * NR], hij[2];
                            V.template load2<decltype(src)::value>(j0, k, e);
#pragma unroll
                            for (int u = 0; u < 2; ++u) hij[u] = -__shfl_sync(0xffffffffu, hs, j0 + u);
                            auto subtract = [&](int u) {
#pragma unroll
                                for (int r = 0; r < NR; r += 2)
                                    fma_pair(w[r], w[r + 1], hij[u], hij[u], e[u * NR + r], e[u * NR + r + 1]);
                            };
                            subtract(0);
                            if (j0 + 1 <= k) subtract(1);
                        });
                        if (NQ == 8 && warp_tail) {
#pragma unroll 4
                            for (int j = 0; j <= k; ++j) {
                                const float hij = __shfl_sync(0xffffffffu, hs, j);
                                const float t0 = tails[j * S.tail + tt[0]], t1 = tails[j * S.tail + tt[1]];
                                w_t[0] = tail[0] ? w_t[0] - hij * t0 : 0.f;
                                w_t[1] = tail[1] ? w_t[1] - hij * t1 : 0.f;
                            }
                        }
                    }
                    float loc3[2] = {0.f, 0.f};
#pragma unroll
                    for (int r = 0; r < NR; ++r) loc3[r & 1] += w[r] * w[r];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (tail[h]) loc3[h] += w_t[h] * w_t[h];
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        loc3[0] += __shfl_xor_sync(0xffffffffu, loc3[0], o);
                        loc3[1] += __shfl_xor_sync(0xffffffffu, loc3[1], o);
                    }
                    if (lane == 0) {
                        norm[(k & 1) * 32 + warp] = loc3[0];
                        norm[(k & 1) * 32 + warp + kGridGroups / 2] = loc3[1];
                    }
                } else if (k > 0) {
                    column(k - 1);
                }
                __syncthreads();
                if (k > 0 && done[(k - 1) & 1]) break;  // the step before was the last
                ++total;
                float s = lane < kGridGroups ? norm[(k & 1) * 32 + lane] : 0.f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (s == 0.f) {  // ||w|| < 1e-30, in FP32
                    if (!rows) column(k);
                    ++k;
                    break;
                }
                if (rows && k + 1 < m) {
                    const float inv_w = grid_inv_sqrt(s);
#pragma unroll
                    for (int r = 0; r < NR; ++r) v[r] = w[r] * inv_w;
                    V.store(k + 1, v);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        v_t[h] = w_t[h] * inv_w;
                        if (tail[h]) tails[(k + 1) * S.tail + tt[h]] = v_t[h];
                    }
                }
                ++k;
            }
            // y from the triangular system; sol += M^-1 V y
            if (!rows) {
                // lane j holds y_j, and column j's entry of the row at hand; one
                // chain of fused products, in order
                double ys = 0.0, rowa = lane < k ? hmat[lane * kGridProjLd + k - 1] : 0.0;
                for (int a = k - 1; a >= 0; --a) {
                    const double row = rowa;
                    if (a > 0 && lane < k) rowa = hmat[lane * kGridProjLd + a - 1];
                    double sum = gvec[a];
                    const double rc = rcp[a], haa = __shfl_sync(0xffffffffu, row, a);
#pragma unroll 4
                    for (int j = a + 1; j < k; ++j)
                        sum -= __shfl_sync(0xffffffffu, row, j) * __shfl_sync(0xffffffffu, ys, j);
                    const double y = fabs(haa) > 1e-30 ? warp_div(sum, haa, rc) : 0.0;
                    if (lane == a) ys = y;
                }
                if (lane < k) yv[lane] = ys;
            }
            __syncthreads();
            if (rows) {
                double* sol = grid_instance_ptrs(L).b;
                double s[NR], s_t[2];
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int p = tid + r * T;
                    s[r] = p < n ? sol[p] : 0.0;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) s_t[h] = tail[h] ? sol[pt + h * T] : 0.0;
                V.template each<2>(k - 1, [&](auto src, auto, int a0) {
                    float e[2 * NR];
                    V.template load2<decltype(src)::value>(a0, k - 1, e);
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (a0 + u < k) {
                            const double y = yv[a0 + u];
                            float z[NR];
                            bool plain = true;
#pragma unroll
                            for (int r = 0; r < NR; ++r) {
                                z[r] = e[u * NR + r] * inv[r];
                                plain = plain && grid_widens(z[r]);
                            }
                            if (plain) {
#pragma unroll
                                for (int r = 0; r < NR; ++r) s[r] += grid_widen(z[r]) * y;
                            } else {
#pragma unroll
                                for (int r = 0; r < NR; ++r) s[r] += f32_to_f64_int(z[r]) * y;
                            }
                            if (NQ == 8 && warp_tail) {
#pragma unroll
                                for (int h = 0; h < 2; ++h)
                                    if (tail[h])
                                        s_t[h] += f32_to_f64_int(tails[(a0 + u) * S.tail + tt[h]] * inv_t[h]) * y;
                            }
                        }
                });
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const int p = tid + r * T;
                    if (p < n) sol[p] = s[r];
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (tail[h]) sol[pt + h * T] = s_t[h];
            }
            __syncthreads();
            if (total >= c.max_krylov) break;
        }
        krylov_total += total;
        // --- Newton update and the reference's convergence test
        bool ok = true, fin = true;
        {
            const double* sol = grid_instance_ptrs(L).b;
            double* x = iterate();
            for (int p = p0; p < n; p += T) {
                const double old = x[p];
                const double nw = old + sol[p];
                const double tl = c.v_reltol * fmax(fabs(nw), fabs(old)) + (p < nn ? c.v_abstol : c.i_abstol);
                ok = ok && fabs(nw - old) <= tl;
                fin = fin && isfinite(nw);
                x[p] = nw;
            }
        }
        ok = __syncthreads_and(ok);
        fin = __syncthreads_and(fin);
        newton_it = it;
        // converged when the step test passes and the KCL residual before this
        // update already met the target
        ok = ok && kept[2] <= c.resid_target;
        if (!fin) {
            status = SP_ST_NONFINITE;
            break;
        }
        if (ok) {
            status = SP_ST_CONVERGED;
            break;
        }
    }
    const double resid = grid_residual<T>(c, grid_instance_ptrs(L), vto(), beta(), iterate(), redd);
    if (tid == 0) {
        const uint32_t i = blockIdx.x;
        L.newton[i] = newton_it;
        L.krylov[i] = krylov_total;
        L.status[i] = status;
        L.resid[i] = resid;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == T / 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kColumns) : "memory");
}

}  // namespace SP_KERNEL_NS
#endif  // SP_KERNEL_NS

}  // namespace sp
