// st_linekern.cuh - the line-operator kernel (compact derivatives, compact
// filter, Gaussian filter) and its launch dispatch, templated on the family:
// CYC = false for the _mf family's bounded lines, CYC = true for periodic
// lines (wrapped halos and the corner correction after the banded solve).
//
// One persistent kernel, k_lines, runs a compile-time list of operations
// ("recipe") on each tile of lines.  A CTA keeps a ring of K slots in shared
// memory; a slot holds the tiles of a recipe's input fields.  The TMA engine
// fills a slot while the CTA's threads solve the slot before it in registers;
// the results overwrite input tiles that no later operation reads and leave
// by TMA stores, or by TMA reductions (cp.reduce, add) where the operation
// accumulates, so the old value never comes to the SM (the reduction keeps
// subnormal floats; measured).  Where only one slot
// fits, its tiles are filled for the next lines one by one, as the operations
// are done with them.
//
// What bounds it: at one field in and one out the TMA ring alone moves 5.5 to
// 5.9 TB/s on 384^3 (x, z and y lines; 0.84 to 0.90 of a plain copy), and an
// accumulation 5.8 to 6.3 TB/s of its 24 bytes per cell.  With the solve, FP64,
// 384^3, against kernels that read the rows from global memory thread by
// thread (about 85 instructions per cell, 512 threads of 64 registers):
//   first derivative x, y, z   187, 166, 178 us (230, 290, 222)
//   filter                     316, 299, 310 us (410, 437, 402)
//   second with first          295, 288, 289 us (490)
//   two first derivatives of Compute_Laplacian in one pass, accumulated
//                              285, 258 us (480 as two passes)
// The solve's latency is what is left: a solve costs about 130 us of a 384^3
// pass, and is hidden only while another CTA of the SM is transferring.
#pragma once
#include <cfloat>
#include <cuda.h>
#include <type_traits>
#include <utility>
#include "st_line.cuh"
#include "st_once.h"

namespace st {

enum OpKind { OP_D1, OP_D2, OP_FILTER, OP_GAUSS, OP_LAP, OP_D1ADD, OP_FILTERM };

// One operation of a recipe: KIND applied to the operand SRC with arguments
// op[ARG]; the result goes to tile OUT (OP_D1ADD: is added to what is there)
// and from there to output field IO (none where IO < 0).
template <int KIND_, class SRC_, int OUT_, int IO_, int ARG_ = IO_>
struct Op {
    static constexpr int KIND = KIND_, OUT = OUT_, IO = IO_, ARG = ARG_;
    using SRC = SRC_;
};
// NIN input fields (tiles 0 .. NIN-1 of a slot), NT tiles of a slot
template <int NIN_, int NT_, class... OPS>
struct Recipe {
    static constexpr int NIN = NIN_, NT = NT_, NOP = sizeof...(OPS);
};

// The recipes (operation order: an operation may overwrite only tiles that no
// later one reads; outputs are indexed as the caller gives them)
using RecD1 = Recipe<1, 1, Op<OP_D1, Src<PR_A, 0>, 0, 0>>;
using RecMul = Recipe<2, 2, Op<OP_D1, Src<PR_MUL, 0, 1>, 0, 0>>;
using RecAddMul = Recipe<3, 3, Op<OP_D1, Src<PR_ADDMUL, 0, 1, 2>, 0, 0>>;
// a b with half the factor, plus c's derivative.  (One derivative of a b / 2 + c
// rounds the sum to the magnitude of c, the pressure, before it is differenced:
// the rms error of the y and z momentum right-hand sides against an extended
// precision grew by 2 to 7 %.)
using RecMulPlus = Recipe<3, 3, Op<OP_D1, Src<PR_MUL, 0, 1>, 0, -1, 1>, Op<OP_D1ADD, Src<PR_A, 2>, 0, 0>>;
using RecD2 = Recipe<1, 1, Op<OP_D2, Src<PR_A, 0>, 0, 0>>;
using RecD2D1 = Recipe<1, 2, Op<OP_D2, Src<PR_A, 0>, 1, 0>, Op<OP_D1, Src<PR_A, 0>, 0, 1>>;
using RecFilter = Recipe<1, 1, Op<OP_FILTER, Src<PR_A, 0>, 0, 0>>;
using RecFilterM = Recipe<1, 1, Op<OP_FILTERM, Src<PR_A, 0>, 0, 0>>;   // the FP32 mode's
using RecGauss = Recipe<1, 1, Op<OP_GAUSS, Src<PR_A, 0>, 0, 0>>;
using RecLap = Recipe<1, 1, Op<OP_LAP, Src<PR_A, 0>, 0, 0>>;
// pairs of first derivatives that share operand fields: outputs 0 and 1
using RecPairA = Recipe<2, 2, Op<OP_D1, Src<PR_MUL, 1, 0>, 1, 1>, Op<OP_D1, Src<PR_A, 0>, 0, 0>>;              // F; U F
using RecPairB = Recipe<3, 3, Op<OP_D1, Src<PR_MULMUL, 0, 1, 2>, 2, 1>, Op<OP_D1, Src<PR_MUL, 0, 1>, 0, 0>>;  // a b; c (a b)
using RecPairC = Recipe<4, 4, Op<OP_D1, Src<PR_SPECT, 0, 1, 2, 3>, 3, 1>, Op<OP_D1, Src<PR_SPEC, 0, 1, 2>, 0, 0>>;
using RecPairD = Recipe<4, 4, Op<OP_D1, Src<PR_MUL, 0, 1>, 0, 0>, Op<OP_D1, Src<PR_ADDMUL, 2, 3, 1>, 2, 1>>;  // a u; (b + c) u
using RecPairE = Recipe<3, 3, Op<OP_D1, Src<PR_MUL, 0, 1>, 0, 0>, Op<OP_D1, Src<PR_MUL, 2, 1>, 2, 1>>;        // a u; b u

template <class T>
struct OpArgT {
    double fac1, fac2;       // first / second derivative factor
    int asym;
    TriTabT<T> t1, t2;       // first / second derivative tables (OP_LAP: t2 the antisymmetric first derivative's)
    unsigned tab, tab2;      // where their copies start in shared memory, from the tables' start
};

template <class T>
struct alignas(64) LineArgsT {
    CUtensorMap in[4], out[2];
    int red[2];                   // output accumulates
    int dir, n, P;
    int jb;                       // x and z lines: tiles along y
    int cblk, ntile;              // tiles per case, in all
    int box;                      // rows of a TMA box (x and z lines)
    int K;                        // slots
    unsigned tb;                  // bytes of a tile
    int *wait_flag;
    OpArgT<T> op[2];
    PenTab p;
    Consts c;
    double k0, k1, k2;
};
using LineArgs = LineArgsT<double>;
using LineArgsF = LineArgsT<float>;

// ---- TMA and mbarrier instructions -----------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Waits for the phase to complete; false if it does not within a second.  (By
// the clock, because how long a poll suspends the thread is the hardware's
// choice, and by polls, so that a kernel which was itself not running for a
// second looks again.)
constexpr unsigned long long kWaitNs = 1000000000ull;
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
    unsigned long long t0 = 0;
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (bar_try(bar, parity)) return true;
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        else if (t - t0 > kWaitNs) return false;
    }
}
__device__ __forceinline__ void tma_load(unsigned dst, const CUtensorMap *m, int c0, int c1, int c2, int c3, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_store(const CUtensorMap *m, int c0, int c1, int c2, int c3, unsigned src, bool red) {
    if (red)
        asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                     ::"l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(src) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];"
                     ::"l"(m), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(src) : "memory");
}
template <int N> __device__ __forceinline__ void wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- the kernel ------------------------------------------------------------
// shared memory: K slots of NT tiles, the carry buffers, the slots' barriers
constexpr int kSlotsMax = 3;
constexpr unsigned kRingBytes = 8u * kSlotsMax + 8u;      // barriers, and the mark of a wait that ran out
template <class V, int L> __host__ __device__ constexpr unsigned corner_bytes() { return 4 * L * sizeof(V); }
// bytes behind the tiles: the carry buffers (two of one value per segment and
// column, or one of two values for the filter), the corner values, the
// barriers and the mark, the filter's outer factors
// (a scan of float carries needs one column more)
template <class V, int L>
__host__ __device__ inline unsigned carry_one(int P) { return (unsigned)(P + (std::is_same<V, F2>::value ? 1 : 0)) * L * (unsigned)sizeof(V); }
template <class V, int L>
__host__ __device__ inline unsigned carry_bytes(int P) { return 2u * carry_one<V, L>(P) + corner_bytes<V, L>() + kRingBytes; }

template <int S, int M, int L, bool YT, bool CYC, class T, class OPD, class Mid>
__device__ __forceinline__ void run_op(const LineArgsT<T> &a, const OpArgT<T> &o, const unsigned char *tabs,
                                       const View<S, L, YT, T> &w, int s, int lane, const CarryT<typename Val<T>::V, L> &cb,
                                       Mid mid) {
    using V = typename Val<T>::V;
    using SRC = typename OPD::SRC;
    const int n = a.n, P = a.P, row0 = s * S;
    auto rd = [&](int i) { return w.template row<SRC>(i); };
    if constexpr (OPD::KIND == OP_D1 || OPD::KIND == OP_D1ADD || OPD::KIND == OP_LAP) {
        V v[S + 4];
        w.template load<SRC, 2>(v);
        rhs_d1<S, CYC>(v, row0, n, o.asym, o.fac1, a.c, rd);
        const T *tab = reinterpret_cast<const T *>(tabs + o.tab);
        tri<S, M, L, CYC>(v, o.t1, tab, s, P, lane, cb, mid);
        w.template store<OPD::KIND == OP_D1ADD>(v, OPD::OUT);
        if constexpr (OPD::KIND == OP_LAP) {
            // the derivative (in the tile now) of a symmetric field is
            // antisymmetric; both passes of Compute_Laplacian in one
            __syncthreads();
            using D = Src<PR_A, OPD::OUT>;
            auto rd2 = [&](int i) { return w.template row<D>(i); };
            w.template load<D, 2>(v);
            rhs_d1<S, CYC>(v, row0, n, 1, o.fac1, a.c, rd2);
            tri<S, M, L, CYC>(v, o.t2, reinterpret_cast<const T *>(tabs + o.tab2), s, P, lane, cb, [] {});
            w.store(v, OPD::OUT);
        }
    } else if constexpr (OPD::KIND == OP_D2) {
        V v[S + 4];
        w.template load<SRC, 2>(v);
        rhs_d2<S, CYC>(v, row0, n, o.asym, o.fac2, a.c, rd);
        tri<S, M, L, CYC>(v, o.t2, reinterpret_cast<const T *>(tabs + o.tab2), s, P, lane, cb, mid);
        w.store(v, OPD::OUT);
    } else if constexpr (OPD::KIND == OP_FILTER || OPD::KIND == OP_FILTERM) {
        V v[S + 8];
        w.template load<SRC, 4>(v);
        rhs_filter<S, CYC>(v, row0, n, o.asym, a.c, rd);
        if constexpr (OPD::KIND == OP_FILTER) pen_solve<S, L>(v, a.p, s, P, lane, cb, mid);
        else pen_solve_m<S / M, M, L>(v, a.p, s, P, lane, cb, mid);
        if constexpr (CYC) cyc_fix<S, L, 4>(v, a.p.cyc + (size_t)s * S * 4, s >= a.p.clo && s < a.p.chi, s, P, lane, cb);
        w.store(v, OPD::OUT);
    } else {
        V v[S + 8];
        w.template load<SRC, 4>(v);
        rhs_gauss<S, CYC>(v, row0, n, a.c, rd);
        __syncthreads();                       // every thread has read its rows
        if (threadIdx.x == 0) mid();
        w.store(v, OPD::OUT);
    }
    proxy_fence();                             // the tile's new values, for the TMA store
}

// What thread 0 needs to know of a recipe: per operation its output tile and
// field, and the input tiles that are free once the operation has read its
// rows (read by no later operation and not written).
template <class R> struct RecipeInfo;
template <int NIN, int NT, class... OPS>
struct RecipeInfo<Recipe<NIN, NT, OPS...>> {
    static constexpr int N = sizeof...(OPS);
    template <class O> __host__ __device__ static constexpr unsigned reads() {
        const int t[4] = {O::SRC::T0, O::SRC::T1, O::SRC::T2, O::SRC::T3};
        unsigned m = 0;
        for (int k = 0; k < O::SRC::n; k++) m |= 1u << t[k];
        return m;
    }
    __host__ __device__ static constexpr int out(int op) { const int o[N] = {OPS::OUT...}; return o[op]; }
    __host__ __device__ static constexpr int io(int op) { const int o[N] = {OPS::IO...}; return o[op]; }
    // TMA store groups of a tile of lines
    __host__ __device__ static constexpr int stores() { int m = 0; for (int k = 0; k < N; k++) m += io(k) >= 0; return m; }
    __host__ __device__ static constexpr unsigned freed(int op) {
        const unsigned rd[N] = {reads<OPS>()...};
        unsigned keep = 0;
        for (int k = 0; k < N; k++) keep |= (k > op ? rd[k] : 0u) | 1u << out(k);
        return rd[op] & ~keep;
    }
};

template <class R> struct RecipeRun;
template <int NIN, int NT, class... OPS>
struct RecipeRun<Recipe<NIN, NT, OPS...>> {
    static constexpr bool uses1(int kind) { return kind == OP_D1 || kind == OP_D1ADD || kind == OP_LAP; }
    static constexpr bool uses2(int kind) { return kind == OP_D2 || kind == OP_LAP; }
    // host: places the operations' tridiagonal tables, returns their bytes
    template <int S, int M, class T>
    static unsigned place_tables(LineArgsT<T> &a) {
        unsigned at = 0;
        auto one = [&](int kind, OpArgT<T> &o) {
            if (uses1(kind)) { o.tab = at; at += tri_bytes(o.t1, a.P * M, S / M, a.P, S); }
            if (uses2(kind)) { o.tab2 = at; at += tri_bytes(o.t2, a.P * M, S / M, a.P, S); }
        };
        (one(OPS::KIND, a.op[OPS::ARG]), ...);
        return at;
    }
    template <int S, int M, class T, class O>
    __device__ __forceinline__ static void fill_one(const LineArgsT<T> &a, unsigned char *tabs) {
        const OpArgT<T> &o = a.op[O::ARG];
        if constexpr (O::KIND == OP_D1 || O::KIND == OP_D1ADD || O::KIND == OP_LAP)
            tri_fill(reinterpret_cast<T *>(tabs + o.tab), o.t1, a.P * M, S / M, a.P, S);
        if constexpr (O::KIND == OP_D2 || O::KIND == OP_LAP)
            tri_fill(reinterpret_cast<T *>(tabs + o.tab2), o.t2, a.P * M, S / M, a.P, S);
    }
    template <int S, int M, class T>
    __device__ __forceinline__ static void fill_tables(const LineArgsT<T> &a, unsigned char *tabs) {
        (fill_one<S, M, T, OPS>(a, tabs), ...);
    }
    // the operations in turn; hook(op) runs in thread 0 behind the first
    // barrier of each
    template <int S, int M, int L, bool YT, bool CYC, class T, class Hook, size_t... Q>
    __device__ __forceinline__ static void run(const LineArgsT<T> &a, const unsigned char *tabs, const View<S, L, YT, T> &w,
                                               int s, int lane,
                                               const CarryT<typename Val<T>::V, L> &cb, Hook hook, std::index_sequence<Q...>) {
        (run_op<S, M, L, YT, CYC, T, OPS>(a, a.op[OPS::ARG], tabs, w, s, lane, cb, [&] { hook(std::integral_constant<int, (int)Q>()); }), ...);
    }
};

template <class R, int S, int M, int L, bool YT, bool CYC, class T>
__global__ void __maxnreg__(80) k_lines(const __grid_constant__ LineArgsT<T> a) {
    using V = typename Val<T>::V;
    using I = RecipeInfo<R>;
    constexpr int W = Val<T>::W, NL = L * W;         // lines of a tile
    constexpr bool PENM = std::is_same<R, RecFilterM>::value, PEN = PENM || std::is_same<R, RecFilter>::value;
    extern __shared__ __align__(1024) unsigned char smem[];
    const unsigned tb = a.tb, slot_b = R::NT * tb;
    const int n = a.n, P = a.P, K = a.K, G = gridDim.x;
    const int tid = threadIdx.x, lane = tid % L, s = tid / L;
    unsigned char *tail = smem + K * slot_b;
    const unsigned cbb = (PENM ? 2u : 1u) * carry_one<V, L>(P * M);
    unsigned char *tab = tail + 2 * cbb + corner_bytes<V, L>() + kRingBytes;
    const CarryT<V, L> cb{reinterpret_cast<V *>(tail), reinterpret_cast<V *>(tail + cbb), reinterpret_cast<V *>(tail + 2 * cbb),
                          reinterpret_cast<const V *>(tab)};
    const unsigned bars = smem_u32(tail + 2 * cbb + corner_bytes<V, L>());
    volatile int *const late = reinterpret_cast<int *>(tail + 2 * cbb + corner_bytes<V, L>() + 8 * kSlotsMax);
    if constexpr (PEN) pen_fill(reinterpret_cast<double *>(tab), a.p, P * M, S / M, !PENM);
    else RecipeRun<R>::template fill_tables<S, M, T>(a, tab);

    // thread 0: transfers of one tile of lines.  x lines: (y, z) at c0, c1
    // and rows along the third coordinate; z lines: (y, x) and rows along the
    // second; y lines: (row in the chunk, line, chunk)
    auto place = [&](int tile, int &c0, int &m, int &cs) {
        if constexpr (YT) { c0 = 0; m = tile * NL; cs = 0; return; }
        cs = tile / a.cblk;
        const int b = tile - cs * a.cblk;
        m = b / a.jb;
        c0 = (b - m * a.jb) * NL;
    };
    auto load_tiles = [&](int tile, int k, unsigned mask) {
        int c0, m, cs;
        place(tile, c0, m, cs);
        const unsigned bar = bars + 8 * k, dst = smem_u32(smem + k * slot_b);
#pragma unroll
        for (int f = 0; f < R::NIN; f++) {
            if (!(mask >> f & 1)) continue;
            if constexpr (YT) tma_load(dst + f * tb, &a.in[f], 0, m, 0, 0, bar);
            else
                for (int r = 0; r < n; r += a.box)
                    tma_load(dst + f * tb + r * 8 * L, &a.in[f], c0, a.dir == 0 ? m : r, a.dir == 0 ? r : m, cs, bar);
        }
    };
    auto expect = [&](int k) { bar_expect(bars + 8 * k, R::NIN * tb); };
    auto store_out = [&](int tile, int k, int op) {
        int c0, m, cs;
        place(tile, c0, m, cs);
        const int io = I::io(op);
        const unsigned src = smem_u32(smem + k * slot_b + I::out(op) * tb);
        if constexpr (YT) tma_store(&a.out[io], 0, m, 0, 0, src, a.red[io] != 0);
        else
            for (int r = 0; r < n; r += a.box)
                tma_store(&a.out[io], c0, a.dir == 0 ? m : r, a.dir == 0 ? r : m, cs, src + r * 8 * L, a.red[io] != 0);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    };
    constexpr unsigned ALL = (1u << R::NIN) - 1;

    if (tid == 0) {
#pragma unroll
        for (int f = 0; f < R::NIN; f++) asm volatile("prefetch.tensormap [%0];" ::"l"(&a.in[f]) : "memory");
#pragma unroll
        for (int f = 0; f < I::stores(); f++) asm volatile("prefetch.tensormap [%0];" ::"l"(&a.out[f]) : "memory");
        for (int k = 0; k < K; k++) bar_init(bars + 8 * k);
        *late = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        proxy_fence();
    }
    __syncthreads();
    pdl_wait();
    if (tid == 0)
        for (int k = 0; k < K; k++)
            if ((int)blockIdx.x + k * G < a.ntile) { expect(k); load_tiles(blockIdx.x + k * G, k, ALL); }

    View<S, L, YT, T> w;
    w.tb = tb; w.lane = lane; w.n = n; w.a = s * S; w.mid = TileAcc<L, YT, T>::start(lane, s * S);
    w.k0 = (typename Val<T>::A)a.k0; w.k1 = (typename Val<T>::A)a.k1; w.k2 = (typename Val<T>::A)a.k2;
    // A wait that runs out ends the CTA: nothing of its tile is stored or
    // loaded, the host reports the flag at the next synchronising call.  Threads
    // may differ about it, so the mark decides: it is written before the first
    // barrier of a tile and read between that and the barrier at its end.  (The
    // end on the mark costs 7 % of the second derivative with the first along y
    // and 1 % elsewhere at most; a barrier that reduces the threads' results
    // instead, or loops that run on without it, cost more.)
    int k = 0, kp = K - 1;          // slot of this tile and of the one before
    unsigned par = 0;
    for (int tile = blockIdx.x; tile < a.ntile; tile += G) {
        if (!bar_wait(bars + 8 * k, par)) {
            *late = 1;
            *reinterpret_cast<volatile int *>(a.wait_flag) = 1;
        }
        w.sm = smem + k * slot_b;
        const int next = tile + (K == 1 ? 1 : K - 1) * G;
        const bool more = next < a.ntile;
        RecipeRun<R>::template run<S, M, L, YT, CYC, T>(a, tab, w, s, lane, cb, [&](auto q) {
            constexpr int OP = decltype(q)::value;
            constexpr bool STORES = OP > 0 && I::io(OP > 0 ? OP - 1 : 0) >= 0;
            if ((STORES || K == 1) && *late) return;
            // the result of the operation before leaves, and with one slot
            // the tiles that are free are filled for the next tile of lines
            if constexpr (STORES) store_out(tile, k, OP - 1);
            if (K == 1 && more) {
                if constexpr (OP == 0) expect(0);
                constexpr unsigned FREED = I::freed(OP);
                if constexpr (FREED != 0) load_tiles(next, 0, FREED);
            }
        }, std::make_index_sequence<I::N>());
        const int dead = *late;
        __syncthreads();
        if (dead) {
            // the slots that loads are in flight to, the tile's own first: the
            // CTA's shared memory has to stay until they have landed
            if (tid == 0)
                for (int j = 0, m = K > 1 && tile >= G ? K - 1 : K; j < m && tile + j * G < a.ntile; j++)
                    bar_wait(bars + 8 * (k + j < K ? k + j : k + j - K), k + j < K ? par : par ^ 1);
            break;
        }
        if (tid == 0) {
            store_out(tile, k, I::N - 1);
            if (K == 1) {
                // the output tiles, as their stores have been read out
                if constexpr (I::stores() == 2) {
                    wait_read<1>();
                    if (more) load_tiles(next, 0, 1u << I::out(0));
                }
                wait_read<0>();
                if (more) load_tiles(next, 0, 1u << I::out(I::N - 1));
            } else {
                // the slot of the tile before, whose stores were issued a
                // whole tile ago
                wait_read<I::stores()>();
                if (tile >= G && more) { expect(kp); load_tiles(next, kp, ALL); }
            }
        }
        kp = k;
        if (++k == K) { k = 0; par ^= 1; }
    }
    pdl_next();
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- launch ------------------------------------------------------------------
// Tensor map of a field whose boxes are (parts of) one tile of nl lines: 4-D
// (y, z, x, case) for x and z lines; (row in a 128-byte chunk, line, chunk)
// with the 128-byte swizzle for y lines
int line_map(st_ctx *c, CUtensorMap *m, const void *p, bool f32, int dir, int nl, int box);

// The dynamic shared memory a kernel may ask for is an attribute of the kernel
// on one device.  It is raised to the device's maximum before the kernel's
// first launch there: a limit that follows the launches' sizes would have to be
// raised again for each, and two threads with contexts of different sizes could
// lower it under each other's launch.
template <auto Kern>
static cudaError_t allow_smem(const st_ctx *c) {
    static OncePerDevice once;   // one mark per kernel instantiation
    return (cudaError_t)once(c->dev, [&] {
        return (int)cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, c->smem_cta);
    });
}

// One launch: fields in[0..NIN-1], outputs out[0..NOUT-1] (a.red set), the
// operations' arguments in a.op; name and bytes for the timing report.
template <class R, int S, int M, int L, bool YT, bool CYC, class T>
static int launch_lines(st_ctx *c, LineArgsT<T> &a, const T *const *in, T *const *out, const char *name) {
    using V = typename Val<T>::V;
    constexpr int NL = L * Val<T>::W;
    const int n = a.n;
    const size_t nlines = c->dm.n3 / (size_t)n;              // lines of one case
    a.cblk = (int)(nlines / NL);
    a.ntile = a.cblk * c->na;
    a.jb = c->dm.n[1] / NL;
    a.box = n <= 256 ? n : n / 2;
    a.wait_flag = c->wait_flag_dev;
    a.tb = (unsigned)n * 8 * L;
    using I = RecipeInfo<R>;
    double fields = R::NIN;
    for (int k = 0; k < R::NIN; k++) {
        ST_TRY(line_map(c, &a.in[k], in[k], sizeof(T) == 4, a.dir, NL, a.box));
    }
    for (int k = 0; k < I::stores(); k++) {
        ST_TRY(line_map(c, &a.out[k], out[k], sizeof(T) == 4, a.dir, NL, a.box));
        fields += a.red[k] ? 2 : 1;
    }
    // Slots and CTAs per SM: two slots or more per CTA, so that a tile's
    // transfers overlap another's solve, in as many CTAs as the registers
    // (80 a thread) and the shared memory hold; one slot in two CTAs where
    // two slots do not fit.
    const unsigned slot = R::NT * a.tb, tail = carry_bytes<V, L>(a.P * M) +
                          (std::is_same<R, RecFilterM>::value ? 2u * carry_one<V, L>(a.P * M) : 0u) +
                          (a.p.id ? pen_bytes(a.p, a.P * M, S / M) : 0u) + RecipeRun<R>::template place_tables<S, M, T>(a);
    const int threads = L * a.P;
    const int by_regs = 65536 / (80 * ((threads + 31) / 32 * 32));
    auto fit = [&](int ctas) { return ((long)(c->smem_sm / ctas) - 1024 - (long)tail) / (long)slot; };   // slots
    int ctas = 1, K = 1;
    const int want = R::NT >= 3 ? 2 : 3;
    for (int q = by_regs < 8 ? by_regs : 8; q >= 1; q--) {
        const long f = fit(q);
        if (f >= 2 || (q == 2 && f == 1 && fit(1) < 3) || q == 1) { ctas = q; K = f > want ? want : (int)f; break; }
    }
    if (K < 1) return fail(c, ST_E_UNSUPPORTED, "line tile does not fit in shared memory");
    a.K = K;
    const size_t smem = (size_t)K * slot + tail;
    long grid = (long)c->sms * ctas;
    if (grid > a.ntile) grid = a.ntile;
    ST_CUDA(c, (allow_smem<k_lines<R, S, M, L, YT, CYC, T>>(c)));
    int pi = prof_start(c, name, fields * sizeof(T) * (double)c->ncell());
    void (*kern)(const LineArgsT<T>) = k_lines<R, S, M, L, YT, CYC, T>;
    const cudaError_t e = launch_pdl(kern, dim3((unsigned)grid), dim3(threads), smem, c->stream, a);
    prof_stop(c, pi);
    ST_CUDA(c, e);
    return ST_OK;
}

// 16 columns where the recipe's tiles fit, 8 otherwise (only recipes of four
// tiles, on lines of more than 432 rows, which have segments of 16 rows)
template <class R, int S, int M, bool CYC, class T>
static int launch_lines_L(st_ctx *c, LineArgsT<T> &a, const T *const *in, T *const *out, const char *name) {
    a.P = a.n / S;
    if constexpr (R::NT == 4 && S == 16 && M == 1) {
        if (4L * 128 * a.n + carry_bytes<typename Val<T>::V, 16>(a.P) + RecipeRun<R>::template place_tables<S, M, T>(a) > c->smem_cta) {
            if (a.dir == 1) return launch_lines<R, S, M, 8, true, CYC, T>(c, a, in, out, name);
            return launch_lines<R, S, M, 8, false, CYC, T>(c, a, in, out, name);
        }
    }
    if (a.dir == 1) return launch_lines<R, S, M, 16, true, CYC, T>(c, a, in, out, name);
    return launch_lines<R, S, M, 16, false, CYC, T>(c, a, in, out, name);
}

// recipe by number
enum RecId { R_D1, R_MUL, R_ADDMUL, R_MULPLUS, R_D2, R_D2D1, R_FILTER, R_GAUSS, R_LAP, R_PAIRA, R_PAIRB, R_PAIRC, R_PAIRD,
             R_PAIRE };

template <int S, int M, bool CYC, class T>
static int launch_rec_S(st_ctx *c, RecId id, LineArgsT<T> &a, const T *const *in, T *const *out) {
    switch (id) {
#define REC(id_, rec_, name_) case id_: return launch_lines_L<rec_, S, M, CYC, T>(c, a, in, out, name_);
        REC(R_D1, RecD1, "k_dfd") REC(R_MUL, RecMul, "k_dfd") REC(R_ADDMUL, RecAddMul, "k_dfd")
        REC(R_MULPLUS, RecMulPlus, "k_dfd")
        REC(R_D2, RecD2, "k_d2fd2") REC(R_D2D1, RecD2D1, "k_d2fd2") REC(R_GAUSS, RecGauss, "k_gauss")
        REC(R_PAIRA, RecPairA, "k_dfd_pair") REC(R_PAIRB, RecPairB, "k_dfd_pair")
        REC(R_PAIRD, RecPairD, "k_dfd_pair") REC(R_PAIRE, RecPairE, "k_dfd_pair")
        case R_FILTER:
            if constexpr (sizeof(T) == 8) return launch_lines_L<RecFilter, S, M, CYC, T>(c, a, in, out, "k_filter");
            break;                    // the compact filter acts on the FP64 state only
        // the species terms and the first-derivative Laplacian exist in the _mf family only
        case R_PAIRC: if constexpr (!CYC) return launch_lines_L<RecPairC, S, M, CYC, T>(c, a, in, out, "k_dfd_pair"); break;
        case R_LAP: if constexpr (!CYC) return launch_lines_L<RecLap, S, M, CYC, T>(c, a, in, out, "k_lap"); break;
#undef REC
    }
    return fail(c, ST_E_UNSUPPORTED, "line operation not available in this mode");
}

// all line-operator launches of one family and type: rows per thread from the
// direction's segments (one per thread for doubles, up to four for floats)
template <bool CYC, class T>
static int launch_rec_t(st_ctx *c, RecId id, LineArgsT<T> &a, const T *const *in, T *const *out) {
    if constexpr (sizeof(T) == 8) {
        if (id == R_FILTER && fp32_mode(c)) {
            switch (c->segf[a.dir]) {
#define SEG(s_, st_, m_) case s_: return launch_lines_L<RecFilterM, st_, m_, CYC, T>(c, a, in, out, "k_filter");
                SEG(2, 8, 4) SEG(3, 12, 4) SEG(4, 16, 4) SEG(6, 12, 2) SEG(8, 16, 2) SEG(12, 12, 1) SEG(16, 16, 1)
#undef SEG
            }
            return fail(c, ST_E_UNSUPPORTED, "unsupported line segmentation");
        }
        return c->seg[a.dir] == 8 ? launch_rec_S<8, 1, CYC, T>(c, id, a, in, out) : launch_rec_S<16, 1, CYC, T>(c, id, a, in, out);
    } else {
        switch (c->segf[a.dir]) {
            case 2: return launch_rec_S<8, 4, CYC, T>(c, id, a, in, out);
            case 3: return launch_rec_S<12, 4, CYC, T>(c, id, a, in, out);
            case 4: return launch_rec_S<16, 4, CYC, T>(c, id, a, in, out);
            case 6: return launch_rec_S<12, 2, CYC, T>(c, id, a, in, out);
            case 8: return launch_rec_S<16, 2, CYC, T>(c, id, a, in, out);
            case 12: return launch_rec_S<12, 1, CYC, T>(c, id, a, in, out);
            default: return launch_rec_S<16, 1, CYC, T>(c, id, a, in, out);
        }
    }
}

// the instantiations, each in its own translation unit: bounded lines
// (st_kernels.cu), periodic lines (st_kernels_cyc.cu), FP32 fields
// (st_kernels_f32.cu) and both (st_kernels_cyc_f32.cu)
int launch_rec(st_ctx *c, RecId id, LineArgs &a, const double *const *in, double *const *out);
int launch_rec_cyc(st_ctx *c, RecId id, LineArgs &a, const double *const *in, double *const *out);
int launch_rec_f32(st_ctx *c, RecId id, LineArgsF &a, const float *const *in, float *const *out);
int launch_rec_cyc_f32(st_ctx *c, RecId id, LineArgsF &a, const float *const *in, float *const *out);

}  // namespace st
