// st_line.cuh - device building blocks of the line operators.
//
// Work decomposition: a CTA owns L neighbouring "columns" of one direction
// (L = 16, or 8 where the tiles of 16 do not fit); a column is one line of
// doubles, or two lines of floats (value type F2), so that a row of L columns
// is 8 L bytes.  The CTA's lines sit in shared memory as tiles that the TMA
// engine loads and stores; thread t works on column t % L and on the rows
// [s S, s S + S) of segment s = t / L, which it holds in registers during a
// solve.  Consequences:
//  - a row of an x or z tile is 128 contiguous bytes, so the threads of half a
//    warp read and write it without bank conflicts, at addresses that differ
//    from the thread's first row by constants (no address arithmetic per row);
//  - a y tile is stored in chunks of 128 bytes along the line, [chunk][line],
//    with the TMA engine's 128-byte swizzle, and read and written 16 bytes
//    (two doubles, four floats) at a time: the same rows of eight neighbouring
//    lines then lie in eight different 16-byte bank groups;
//  - segments exchange their end values through shared memory once per
//    recurrence direction; boundary rows belong to the first and last
//    segments only.
#pragma once
#include <type_traits>
#include "st_internal.h"

namespace st {

// two float lines at one row
struct F2 {
    float x, y;
    F2() = default;
    __host__ __device__ constexpr F2(float a, float b) : x(a), y(b) {}
    __host__ __device__ F2(double v) : x((float)v), y((float)v) {}   // a constant on both lines
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return F2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-a.x, -a.y); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ F2 operator*(F2 a, float k) { return F2(a.x * k, a.y * k); }
__device__ __forceinline__ F2 operator*(double k, F2 a) { return F2((float)k * a.x, (float)k * a.y); }
__device__ __forceinline__ F2 operator*(F2 a, double k) { return a * (float)k; }
// k*b + c with one rounding (the solves' explicit fma)
__device__ __forceinline__ double vfma(double k, double b, double c) { return fma(k, b, c); }
__device__ __forceinline__ F2 vfma(float k, F2 b, F2 c) { return F2(fmaf(k, b.x, c.x), fmaf(k, b.y, c.y)); }

// storage type T -> value type V of a column, its scalar A, lines per column W
template <class T> struct Val;
template <> struct Val<double> { using V = double; using A = double; static constexpr int W = 1; };
template <> struct Val<float> { using V = F2; using A = float; static constexpr int W = 2; };

// ---- tile access -----------------------------------------------------------
// Rows of a thread's column are read in units of E rows, whose values come
// with one shared-memory access per line.  Offsets are bytes from the tile's
// start: start(lane, row) of the unit of a row, unit(start, q) of the row q
// behind it (q a multiple of E and a constant; y lines: within the chunk, and
// no carry between the unit numbers: a start row that is a multiple of 16 with
// q < 16, or of 8 with q < 8).
template <int L, bool YT, class T> struct TileAcc;

template <int L, class T> struct TileAcc<L, false, T> {          // x and z lines: [row][column]
    using V = typename Val<T>::V;
    static constexpr int E = 1;
    __device__ __forceinline__ static unsigned start(int lane, int row) { return 8u * lane + 8u * L * row; }
    __device__ __forceinline__ static unsigned unit(unsigned s, int q) { return s + 8u * L * q; }
    __device__ __forceinline__ static void get(V (&w)[1], const unsigned char *p) { w[0] = *reinterpret_cast<const V *>(p); }
    __device__ __forceinline__ static void put(unsigned char *p, const V *w) { *reinterpret_cast<V *>(p) = w[0]; }
    __device__ __forceinline__ static V one(const unsigned char *t, int lane, int row) {
        return *reinterpret_cast<const V *>(t + start(lane, row));
    }
};
// y lines: the 16-byte unit u of line l's chunk c is at ((c NL + l) 8 + (u ^ l % 8)) 16
template <int L, class T> struct TileAccY {
    static constexpr int NL = L * Val<T>::W, RC = 128 / (int)sizeof(T), E = 16 / (int)sizeof(T);
    __device__ __forceinline__ static unsigned start(int lane, int row) {
        return (unsigned)(row / RC) * (NL * 128u) + 128u * lane + (((unsigned)(row % RC / E) ^ (lane & 7u)) << 4);
    }
    __device__ __forceinline__ static unsigned unit(unsigned s, int q) { return s ^ ((unsigned)(q / E) << 4); }
};
template <int L> struct TileAcc<L, true, double> : TileAccY<L, double> {
    using B = TileAccY<L, double>;
    __device__ __forceinline__ static void get(double (&w)[2], const unsigned char *p) {
        const double2 d = *reinterpret_cast<const double2 *>(p);
        w[0] = d.x; w[1] = d.y;
    }
    __device__ __forceinline__ static void put(unsigned char *p, const double *w) {
        *reinterpret_cast<double2 *>(p) = make_double2(w[0], w[1]);
    }
    __device__ __forceinline__ static double one(const unsigned char *t, int lane, int row) {
        return *reinterpret_cast<const double *>(t + B::start(lane, row) + 8 * (row & 1));
    }
};
template <int L> struct TileAcc<L, true, float> : TileAccY<L, float> {   // the column's lines: lane and lane + L
    using B = TileAccY<L, float>;
    static constexpr unsigned SECOND = L * 128u;
    __device__ __forceinline__ static void get(F2 (&w)[4], const unsigned char *p) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + SECOND);
        w[0] = F2(a.x, b.x); w[1] = F2(a.y, b.y); w[2] = F2(a.z, b.z); w[3] = F2(a.w, b.w);
    }
    __device__ __forceinline__ static void put(unsigned char *p, const F2 *w) {
        *reinterpret_cast<float4 *>(p) = make_float4(w[0].x, w[1].x, w[2].x, w[3].x);
        *reinterpret_cast<float4 *>(p + SECOND) = make_float4(w[0].y, w[1].y, w[2].y, w[3].y);
    }
    __device__ __forceinline__ static F2 one(const unsigned char *t, int lane, int row) {
        const unsigned char *p = t + B::start(lane, row) + 4 * (row & 3);
        return F2(*reinterpret_cast<const float *>(p), *reinterpret_cast<const float *>(p + SECOND));
    }
};

// ---- producer expressions --------------------------------------------------
// number of fields an expression reads, and its value
template <int OP> constexpr int prod_n = OP == PR_A ? 1 : OP == PR_MUL ? 2 : OP == PR_SPECT ? 4 : 3;
template <int OP, class V, class A>
__device__ __forceinline__ V prod_val(V a, V b, V c, V d, A k0, A k1, A k2) {
    if constexpr (OP == PR_MUL) return a * b;
    else if constexpr (OP == PR_ADDMUL) return (a + b) * c;
    else if constexpr (OP == PR_MULMUL) return c * (a * b);
    else if constexpr (OP == PR_SPEC) return a * b * c + a * c * k0 * k1;
    else if constexpr (OP == PR_SPECT) { V fl = a * b * c + a * c * k0 * k1; return k2 * d * fl; }
    else return a;
}

// The operand of one operation: a producer expression of the tiles I0..I3 of
// the current slot.
template <int OP, int I0 = 0, int I1 = 0, int I2 = 0, int I3 = 0>
struct Src {
    static constexpr int op = OP, n = prod_n<OP>, T0 = I0, T1 = I1, T2 = I2, T3 = I3;
    __device__ static constexpr int tile(int k) { return k == 0 ? I0 : k == 1 ? I1 : k == 2 ? I2 : I3; }
};

// One thread's view of the slot's tiles
template <int S, int L, bool YT, class T>
struct View {
    using V = typename Val<T>::V;
    using A = typename Val<T>::A;
    using Acc = TileAcc<L, YT, T>;
    unsigned char *sm;        // slot's first tile
    unsigned tb;              // bytes of a tile
    int lane, n, a;           // column, rows of the line, first row of the segment
    unsigned mid;             // start of row a
    A k0, k1, k2;             // producer constants

    // offset of the unit of row a + q
    __device__ __forceinline__ unsigned own(int q) const {
        if constexpr (YT && S % 8 != 0) return Acc::start(lane, a + q);
        else return Acc::unit(mid, q);
    }
    template <class SRC>
    __device__ __forceinline__ V row(int i) const {               // one row (boundary closures)
        V x[4];
#pragma unroll
        for (int k = 0; k < SRC::n; k++) x[k] = Acc::one(sm + SRC::tile(k) * tb, lane, i);
        return prod_val<SRC::op, V, A>(x[0], x[1], x[2], x[3], k0, k1, k2);
    }
    // rows a-H .. a+S+H-1 into v; the rows before the line are the last rows
    // of it and those behind it its first ones (what a periodic line wants;
    // bounded lines overwrite every value that such a row enters)
    template <class SRC, int H>
    __device__ __forceinline__ void load(V (&v)[S + 2 * H]) const {
        constexpr int E = Acc::E, HA = (H + E - 1) / E * E;        // halo in whole units
        const unsigned lo = Acc::start(lane, (a == 0 ? n : a) - HA), hi = Acc::start(lane, a + S == n ? 0 : a + S);
#pragma unroll
        for (int q = 0; q < S + 2 * HA; q += E) {
            const unsigned o = q < HA ? Acc::unit(lo, q) : q < S + HA ? own(q - HA) : Acc::unit(hi, q - S - HA);
            V x[4][E];
#pragma unroll
            for (int k = 0; k < SRC::n; k++) Acc::get(x[k], sm + SRC::tile(k) * tb + o);
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int r = q + e - (HA - H);
                if (r >= 0 && r < S + 2 * H)
                    v[r] = prod_val<SRC::op, V, A>(x[0][e], SRC::n > 1 ? x[1][e] : V(), SRC::n > 2 ? x[2][e] : V(),
                                                   SRC::n > 3 ? x[3][e] : V(), k0, k1, k2);
            }
        }
    }
    // ADD: the sum of the tile's value and r
    template <bool ADD = false, int N>
    __device__ __forceinline__ void store(V (&r)[N], int t) const {
        unsigned char *p = sm + t * tb;
#pragma unroll
        for (int q = 0; q < S; q += Acc::E) {
            if constexpr (ADD) {
                V x[Acc::E];
                Acc::get(x, p + own(q));
#pragma unroll
                for (int e = 0; e < Acc::E; e++) r[q + e] = x[e] + r[q + e];
            }
            Acc::put(p + own(q), &r[q]);
        }
    }
};

// ---- carry exchange --------------------------------------------------------
// Shared buffers of a solve: each segment's end value(s) per column.
template <class V, int L>
struct CarryT {
    V *a, *b;                 // [segment][L] end values, forward and backward
    V *cy;                    // [4][L] corner values of periodic lines
    const V *tab;             // filter: the factors of the rows outside the constant range
};

// ---- tridiagonal tables in shared memory -----------------------------------
// What a solve reads besides the constants of the interior segments: the
// factors and responses of the other segments' rows, the carry weights, the
// corner correction of periodic lines and the float solves' scan factors.
// A CTA copies them once, before it waits for the kernel before it: loads from
// global memory in the solve would each stand in its dependent chain (a first
// derivative at 64^3 took 8.0 us with them and a Gaussian pass, which has
// none, 4.5).
constexpr int kTriRow = 5;           // double: -l, g, id, -(up id), h; float: l, g, id, up, h
constexpr int kScanSteps = 5;        // log2(kMaxSeg)
template <class A> __host__ __device__ __forceinline__ int tri_outer(const TriTabT<A> &T, int P) { return T.slo + (P - T.shi); }
template <class A> __host__ __device__ __forceinline__ bool tri_scan(const TriTabT<A> &T) {
    return sizeof(A) == 4 && (T.kf > 2 * kScanSteps || T.kb > 2 * kScanSteps);
}
// P, S: segments and rows of the solve; Pc, Sc: of the corner correction (the
// kernel's threads)
template <class A> __host__ __device__ __forceinline__ unsigned tri_bytes(const TriTabT<A> &T, int P, int S, int Pc, int Sc) {
    unsigned v = tri_outer(T, P) * S * kTriRow + (tri_scan(T) ? 2 * kScanSteps * kMaxSeg : (T.kf + T.kb) * P);
    if (T.cyc) v += (T.clo + (Pc - T.chi)) * Sc * 2;
    return (v * (unsigned)sizeof(A) + 15u) & ~15u;
}
template <class A> struct TriSm {
    const A *row, *wf, *wb, *cyc;    // scan: wf, wb the scan factors
    __device__ __forceinline__ TriSm(const A *base, const TriTabT<A> &T, int P, int S) {
        row = base;
        wf = row + tri_outer(T, P) * S * kTriRow;
        wb = wf + (tri_scan(T) ? kScanSteps * kMaxSeg : T.kf * P);
        cyc = wb + (tri_scan(T) ? kScanSteps * kMaxSeg : T.kb * P);
    }
};
template <class A> __device__ inline void tri_fill(A *base, const TriTabT<A> &T, int P, int S, int Pc, int Sc) {
    const TriSm<A> m(base, T, P, S);
    const int no = tri_outer(T, P) * S;
    for (int q = threadIdx.x; q < no; q += blockDim.x) {
        const int o = q / S, i = (o < T.slo ? o : o - T.slo + T.shi) * S + q % S;
        A *d = base + q * kTriRow;
        const A l = T.l[i], id = T.id[i], up = T.up[i];
        d[0] = sizeof(A) == 8 ? -l : l;
        d[1] = T.g[i];
        d[2] = id;
        d[3] = sizeof(A) == 8 ? -(up * id) : up;
        d[4] = T.h[i];
    }
    A *wf = const_cast<A *>(m.wf), *wb = const_cast<A *>(m.wb), *cy = const_cast<A *>(m.cyc);
    if (tri_scan(T)) {
        for (int q = threadIdx.x; q < kScanSteps * kMaxSeg; q += blockDim.x) { wf[q] = T.sf[q]; wb[q] = T.sb[q]; }
    } else {                          // [distance - 1][segment]
        for (int q = threadIdx.x; q < T.kf * P; q += blockDim.x) {
            const int d = q / P + 1, s = q % P;
            wf[q] = s >= d ? T.wf[(s - d) * P + s] : (A)0;
        }
        for (int q = threadIdx.x; q < T.kb * P; q += blockDim.x) {
            const int d = q / P + 1, s = q % P;
            wb[q] = s + d < P ? T.wb[(s + d) * P + s] : (A)0;
        }
    }
    if (T.cyc) {
        const int nc = (T.clo + (Pc - T.chi)) * Sc * 2;
        for (int q = threadIdx.x; q < nc; q += blockDim.x) {
            const int o = q / (2 * Sc), s = o < T.clo ? o : o - T.clo + T.chi;
            cy[q] = T.cyc[(size_t)s * Sc * 2 + q % (2 * Sc)];
        }
    }
}

// ---- periodic lines: corner correction after the banded solve ------------
// x_i = y_i - sum_k K_ik y_{j_k} with the corner rows j = {0, n-1} (K = 2,
// tridiagonal) or {0, 1, n-2, n-1} (K = 4, pentadiagonal); the table holds
// -K row-major, here of the thread's rows.  The first and last segments
// publish the corner values.  K decays away from the ends: segments whose
// weights are all below 1e-22 (skip) keep their values.
template <int S, int L, int KC, int N, class V, class A>
__device__ __forceinline__ void cyc_fix(V (&r)[N], const A *kr, bool skip, int s, int P, int lane, const CarryT<V, L> &cb) {
    if (KC == 2) {
        if (s == 0) cb.cy[lane] = r[0];
        if (s == P - 1) cb.cy[L + lane] = r[S - 1];
    } else {
        if (s == 0) { cb.cy[lane] = r[0]; cb.cy[L + lane] = r[1]; }
        if (s == P - 1) { cb.cy[2 * L + lane] = r[S - 2]; cb.cy[3 * L + lane] = r[S - 1]; }
    }
    __syncthreads();
    if (skip) return;
    V y[KC];
#pragma unroll
    for (int k = 0; k < KC; k++) y[k] = cb.cy[k * L + lane];
#pragma unroll
    for (int t = 0; t < S; t++) {
        V v = r[t];
#pragma unroll
        for (int k = 0; k < KC; k++) v = vfma(kr[t * KC + k], y[k], v);
        r[t] = v;
    }
}
template <int S, int L, int N, class V, class A>
__device__ __forceinline__ void cyc_tri(V (&r)[N], const TriTabT<A> &T, const A *tab, int Ps, int Ss, int s, int P, int lane,
                                        const CarryT<V, L> &cb) {
    const TriSm<A> m(tab, T, Ps, Ss);
    cyc_fix<S, L, 2>(r, m.cyc + (s < T.clo ? s : s - T.chi + T.clo) * (2 * S), s >= T.clo && s < T.chi, s, P, lane, cb);
}

// ---- segmented constant-coefficient tridiagonal solve --------------------
// Forward elimination r'_i = r_i - l_i r'_{i-1} and back substitution
// x_i = (r'_i - c_i x_{i+1}) / (b'_i + tiny) of tridiagonal_serial
// (src/tridiagonal.f90:274-284) per segment with zero carries, then the
// carries: each segment sums the few segments before it (after it) whose
// weight can still change a result, and adds its rows' responses.  The
// sweeps are explicit fmas (one rounding per step).  Away from the line's
// ends (segments slo <= s < shi) the factors are constants, which come from
// the kernel parameters and need no loads; the responses there are the same
// in every segment.  tab: the tables in shared memory (tri_fill).
// Buffers: the caller has a barrier between this solve's first write of cb.a
// and the previous solve's last read of it (the barrier after its cb.b
// exchange is one).
// mid: what thread 0 does once every thread has read its rows (behind the
// first barrier).
template <int S, int L, int N, class V, class A, class Mid>
__device__ __forceinline__ void tri_solve(V (&r)[N], const TriTabT<A> &T, const A *tab, int s, int P, int lane,
                                          const CarryT<V, L> &cb, Mid mid) {
    const TriSm<A> m(tab, T, P, S);
    const bool flat = s >= T.slo && s < T.shi;
    const A *row = m.row + (s < T.slo ? s : s - T.shi + T.slo) * (S * kTriRow);
    if (flat) {
        const A l = -T.cl;
#pragma unroll
        for (int t = 1; t < S; t++) r[t] = vfma(l, r[t - 1], r[t]);
    } else {
#pragma unroll
        for (int t = 1; t < S; t++) r[t] = vfma(row[t * kTriRow], r[t - 1], r[t]);
    }
    cb.a[s * L + lane] = r[S - 1];
    __syncthreads();
    if (threadIdx.x == 0) mid();
    V cin = V(0.0);
#pragma unroll 4
    for (int d = min(s, T.kf); d > 0; d--) cin = vfma(m.wf[(d - 1) * P + s], cb.a[(s - d) * L + lane], cin);
    if (flat) {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = vfma(T.cg[t], cin, r[t]);
        const A id = T.cid, ui = -(T.cup * T.cid);
        r[S - 1] = r[S - 1] * id;
#pragma unroll
        for (int t = S - 2; t >= 0; t--) r[t] = vfma(ui, r[t + 1], r[t] * id);
    } else {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = vfma(row[t * kTriRow + 1], cin, r[t]);
        r[S - 1] = r[S - 1] * row[(S - 1) * kTriRow + 2];
#pragma unroll
        for (int t = S - 2; t >= 0; t--) r[t] = vfma(row[t * kTriRow + 3], r[t + 1], r[t] * row[t * kTriRow + 2]);
    }
    cb.b[s * L + lane] = r[0];
    __syncthreads();
    V ein = V(0.0);
#pragma unroll 4
    for (int d = 1, de = min(P - 1 - s, T.kb); d <= de; d++) ein = vfma(m.wb[(d - 1) * P + s], cb.b[(s + d) * L + lane], ein);
    if (flat) {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = vfma(T.ch[t], ein, r[t]);
    } else {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = vfma(row[t * kTriRow + 4], ein, r[t]);
    }
}

// ---- the FP32 mode's tridiagonal solve --------------------------------------
// The float solve keeps its own segmentation (S rows, P M segments of a line)
// and rounding (products and sums of the sweeps not fused): single-precision
// results depend on both through the fourth differences of the artificial
// viscosity, and stay what they are.  A thread works on M consecutive
// segments.  Carries that reach further than ten segments (short lines) come
// from a scan of the affine recurrence, one warp per column with shuffles.
__device__ __forceinline__ F2 shfl_seg(bool up, F2 v, int d) {
    return F2(up ? __shfl_up_sync(0xffffffffu, v.x, d) : __shfl_down_sync(0xffffffffu, v.x, d),
              up ? __shfl_up_sync(0xffffffffu, v.y, d) : __shfl_down_sync(0xffffffffu, v.y, d));
}
// buf[column (P + 1) + segment]: inclusive scan f(s) = a(s) + t_k(s) f(s - 2^k)
// (FWD) or g(s) = b(s) + u_k(s) g(s + 2^k), with the products of 2^k
// consecutive transfer factors in [kScanSteps][kMaxSeg] tables
template <int L, bool FWD>
__device__ __forceinline__ void seg_scan_warp(F2 *buf, const float *tab, int P) {
    const int l = threadIdx.x & 31, nw = blockDim.x >> 5;
    if ((int)(threadIdx.x >> 5) >= nw) return;     // a half warp takes no column
    for (int ln = threadIdx.x >> 5; ln < L; ln += nw) {
        F2 *row = buf + ln * (P + 1);
        F2 f = l < P ? row[l] : F2(0.0);
        for (int k = 0, d = 1; d < P; k++, d <<= 1) {
            const F2 o = shfl_seg(FWD, f, d);
            if (FWD ? (l >= d && l < P) : (l + d < P)) f = vfma(tab[k * kMaxSeg + l], o, f);
        }
        if (l < P) row[l] = f;
    }
}
template <int S, int M, int L, int N, class Mid>
__device__ __forceinline__ void tri_solve_f(F2 (&r)[N], const TriTabT<float> &T, const float *tab, int s, int Pt, int lane,
                                            const CarryT<F2, L> &cb, Mid mid) {
    const int P = Pt * M, s0 = s * M;
    const bool scan = tri_scan(T);
    const TriSm<float> sm(tab, T, P, S);
    auto outer = [&](int q) { return sm.row + (q < T.slo ? q : q - T.shi + T.slo) * (S * kTriRow); };
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 1; t < S; t++) r[o + t] = r[o + t] - r[o + t - 1] * T.cl;
        } else {
            const float *row = outer(q);
#pragma unroll
            for (int t = 1; t < S; t++) r[o + t] = r[o + t] - r[o + t - 1] * row[t * kTriRow];
        }
        if (scan) cb.a[lane * (P + 1) + q] = r[o + S - 1];
        else cb.a[q * L + lane] = r[o + S - 1];
    }
    __syncthreads();
    if (threadIdx.x == 0) mid();
    if (scan) {
        seg_scan_warp<L, true>(cb.a, sm.wf, P);
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        F2 cin = F2(0.0);
        if (scan) {
            if (q > 0) cin = cb.a[lane * (P + 1) + q - 1];
        } else {
#pragma unroll 4
            for (int d = min(q, T.kf); d > 0; d--) cin = vfma(sm.wf[(d - 1) * P + q], cb.a[(q - d) * L + lane], cin);
        }
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = vfma(T.cg[t], cin, r[o + t]);
            r[o + S - 1] = r[o + S - 1] * T.cid;
#pragma unroll
            for (int t = S - 2; t >= 0; t--) r[o + t] = (r[o + t] - r[o + t + 1] * T.cup) * T.cid;
        } else {
            const float *row = outer(q);
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = vfma(row[t * kTriRow + 1], cin, r[o + t]);
            r[o + S - 1] = r[o + S - 1] * row[(S - 1) * kTriRow + 2];
#pragma unroll
            for (int t = S - 2; t >= 0; t--) r[o + t] = (r[o + t] - r[o + t + 1] * row[t * kTriRow + 3]) * row[t * kTriRow + 2];
        }
        if (scan) cb.b[lane * (P + 1) + q] = r[o];
        else cb.b[q * L + lane] = r[o];
    }
    __syncthreads();
    if (scan) {
        seg_scan_warp<L, false>(cb.b, sm.wb, P);
        __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        F2 ein = F2(0.0);
        if (scan) {
            if (q + 1 < P) ein = cb.b[lane * (P + 1) + q + 1];
        } else {
#pragma unroll 4
            for (int d = 1, de = min(P - 1 - q, T.kb); d <= de; d++)
                ein = vfma(sm.wb[(d - 1) * P + q], cb.b[(q + d) * L + lane], ein);
        }
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = vfma(T.ch[t], ein, r[o + t]);
        } else {
            const float *row = outer(q);
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = vfma(row[t * kTriRow + 4], ein, r[o + t]);
        }
    }
}
// the solve of a field type (S rows per thread, in M segments for floats) and,
// on periodic lines, the corner correction
template <int S, int M, int L, bool CYC, int N, class V, class A, class Mid>
__device__ __forceinline__ void tri(V (&r)[N], const TriTabT<A> &T, const A *tab, int s, int P, int lane, const CarryT<V, L> &cb,
                                    Mid mid) {
    if constexpr (sizeof(A) == 4) tri_solve_f<S / M, M, L>(r, T, tab, s, P, lane, cb, mid);
    else tri_solve<S, L>(r, T, tab, s, P, lane, cb, mid);
    if constexpr (CYC) cyc_tri<S, L>(r, T, tab, P * M, S / M, s, P, lane, cb);
}

// The factors of the rows outside the constant range sit in shared memory
// (kPenRow doubles a row; the L1 cache is left with what the tiles do not
// take, and loads that miss it would stand in the recurrences' chains),
// followed by the outer segments' transfer matrices.
constexpr int kPenRow = 9;           // p1, p2, g1, g2, id, id q1, id q2, h1, h2
__host__ __device__ __forceinline__ int pen_outer(const PenTab &T, int P) { return T.slo + (P - T.shi); }   // segments
__host__ __device__ __forceinline__ unsigned pen_bytes(const PenTab &T, int P, int S) {
    return (unsigned)pen_outer(T, P) * (S * kPenRow + 8) * 8u;
}
// fused: as the fmas of pen_solve take them (negated, the back substitution's
// times id), with the transfer matrices; otherwise as they are
__device__ inline void pen_fill(double *tab, const PenTab &T, int P, int S, bool fused) {
    const int no = pen_outer(T, P);
    for (int q = threadIdx.x; q < no * S; q += blockDim.x) {
        const int o = q / S, s = o < T.slo ? o : o - T.slo + T.shi, i = s * S + q % S;
        double *d = tab + q * kPenRow;
        const double id = T.id[i];
        d[0] = fused ? -T.p1[i] : T.p1[i]; d[1] = fused ? -T.p2[i] : T.p2[i];
        d[2] = T.g1[i]; d[3] = T.g2[i]; d[4] = id;
        d[5] = fused ? -(T.q1[i] * id) : T.q1[i]; d[6] = fused ? -(T.q2[i] * id) : T.q2[i];
        d[7] = T.h1[i]; d[8] = T.h2[i];
    }
    if (!fused) return;
    for (int q = threadIdx.x; q < no * 8; q += blockDim.x) {
        const int o = q / 8, s = o < T.slo ? o : o - T.slo + T.shi;
        tab[no * S * kPenRow + q] = q % 8 < 4 ? T.sf[4 * s + q % 8] : T.sb[4 * s + q % 8 - 4];
    }
}

// The carry recurrence over the segments, one column per thread: on entry
// buf holds each segment's end values, on exit its carry-in.  Forward
// f(s) = a(s) + M_s f(s-1), backward g(s) = b(s) + N_s g(s+1).  The next
// segment's values are fetched while the one before is worked on; the chain
// is two fmas per segment.
template <int L, bool FWD>
__device__ __forceinline__ void pen_scan(double *buf, const double *mat, const double (&mc)[4], int slo, int shi, int P, int lane) {
    const int PL = P * L, step = FWD ? L : -L;
    double *p = buf + (FWD ? 0 : (P - 1) * L) + lane;
    double f1 = 0.0, f2 = 0.0, x1 = p[0], x2 = p[PL];
#pragma unroll 2
    for (int k = 0; k < P; k++, p += step) {
        const int q = FWD ? k : P - 1 - k;
        double y1 = 0.0, y2 = 0.0;
        if (k + 1 < P) { y1 = p[step]; y2 = p[PL + step]; }
        p[0] = f1;
        p[PL] = f2;
        double n1;
        if (q >= slo && q < shi) {
            n1 = fma(mc[0], f1, fma(mc[1], f2, x1));
            f2 = fma(mc[2], f1, fma(mc[3], f2, x2));
        } else {
            const double *m = mat + 8 * (q < slo ? q : q - shi + slo);
            n1 = fma(m[0], f1, fma(m[1], f2, x1));
            f2 = fma(m[2], f1, fma(m[3], f2, x2));
        }
        f1 = n1;
        x1 = y1; x2 = y2;
    }
}

// ---- segmented constant-coefficient pentadiagonal solve ------------------
// Elimination order of pentadiagonal_serial (src/pentadiagonal.f90:340-372):
// r'_i = (r_i - k2 r'_{i-2}) - k1 r'_{i-1};  x_i = ((r'_i - D'_i x_{i+1})
// - E_i x_{i+2}) / (C'_i + tiny).  Carries are 2-vectors that reach over most
// of the line (the system is nearly singular), so one warp runs the carry
// recurrence over the segments, one thread per column, between two barriers,
// and every segment then picks up its carry.  (The FP32 mode's filter keeps a
// scan by all threads, log2(P) steps with a barrier each: 384^3 runs at 0.45 of
// a plain copy with either.)
// Buffer: cb.a is [2][segment][L] and serves both directions (a thread reads
// and writes its own segment's entry; only the scanning warp touches others,
// between barriers).
template <int S, int L, int N, class Mid>
__device__ __forceinline__ void pen_solve(double (&r)[N], const PenTab &T, int s, int P, int lane,
                                          const CarryT<double, L> &cb, Mid mid) {
    const int PL = P * L, at = s * L + lane;
    const bool flat = s >= T.slo && s < T.shi;
    const double *tab = cb.tab + (s < T.slo ? s : s - T.shi + T.slo) * (S * kPenRow);
    const double *mat = cb.tab + pen_outer(T, P) * (S * kPenRow);
    if (flat) {
        const double p1 = -T.cp1, p2 = -T.cp2;
        r[1] = fma(p1, r[0], r[1]);
#pragma unroll
        for (int t = 2; t < S; t++) r[t] = fma(p1, r[t - 1], fma(p2, r[t - 2], r[t]));
    } else {
        r[1] = fma(tab[kPenRow], r[0], r[1]);
#pragma unroll
        for (int t = 2; t < S; t++) r[t] = fma(tab[t * kPenRow], r[t - 1], fma(tab[t * kPenRow + 1], r[t - 2], r[t]));
    }
    cb.a[at] = r[S - 1];
    cb.a[PL + at] = r[S - 2];
    __syncthreads();
    if (threadIdx.x < L) pen_scan<L, true>(cb.a, mat, T.cm, T.slo, T.shi, P, lane);
    if (threadIdx.x == 0) mid();
    __syncthreads();
    {
        const double c1 = cb.a[at], c2 = cb.a[PL + at];
        if (flat) {
#pragma unroll
            for (int t = 0; t < S; t++) r[t] = fma(T.cg1[t], c1, fma(T.cg2[t], c2, r[t]));
            const double id = T.cid, q1 = -(T.cq1 * T.cid), q2 = -(T.cq2 * T.cid);
            r[S - 1] = r[S - 1] * id;
            r[S - 2] = fma(q1, r[S - 1], r[S - 2] * id);
#pragma unroll
            for (int t = S - 3; t >= 0; t--) r[t] = fma(q1, r[t + 1], fma(q2, r[t + 2], r[t] * id));
        } else {
#pragma unroll
            for (int t = 0; t < S; t++) r[t] = fma(tab[t * kPenRow + 2], c1, fma(tab[t * kPenRow + 3], c2, r[t]));
            r[S - 1] = r[S - 1] * tab[(S - 1) * kPenRow + 4];
            r[S - 2] = fma(tab[(S - 2) * kPenRow + 5], r[S - 1], r[S - 2] * tab[(S - 2) * kPenRow + 4]);
#pragma unroll
            for (int t = S - 3; t >= 0; t--)
                r[t] = fma(tab[t * kPenRow + 5], r[t + 1], fma(tab[t * kPenRow + 6], r[t + 2], r[t] * tab[t * kPenRow + 4]));
        }
    }
    cb.a[at] = r[0];
    cb.a[PL + at] = r[1];
    __syncthreads();
    if (threadIdx.x < L) pen_scan<L, false>(cb.a, mat + 4, T.cn, T.slo, T.shi, P, lane);
    __syncthreads();
    const double e1 = cb.a[at], e2 = cb.a[PL + at];
    if (flat) {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = fma(T.ch1[t], e1, fma(T.ch2[t], e2, r[t]));
    } else {
#pragma unroll
        for (int t = 0; t < S; t++) r[t] = fma(tab[t * kPenRow + 7], e1, fma(tab[t * kPenRow + 8], e2, r[t]));
    }
}

// The FP32 mode's state filter keeps its own segmentation and rounding, as its
// float solves do (a last-bit change of the state can round a float copy of it
// the other way, which the fourth differences then magnify): unfused sweeps,
// factors in double, and the carries by a scan f(s) = a(s) + M_s f(s-1) over
// the segments in log2 steps by all threads over a double buffer.  A thread
// works on M consecutive segments of S rows; the factors of the rows outside
// the constant range are in shared memory (pen_fill).
template <int S, int M, int L, int N, class Mid>
__device__ __forceinline__ void pen_solve_m(double (&r)[N], const PenTab &T, int s, int Pt, int lane, const CarryT<double, L> &cb,
                                            Mid mid) {
    const int P = Pt * M, s0 = s * M, PL = P * L;
    auto outer = [&](int q) { return cb.tab + (q < T.slo ? q : q - T.shi + T.slo) * (S * kPenRow); };
    double f1[M], f2[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 1; t < S; t++) {
                double v = r[o + t];
                if (t >= 2) v = v - T.cp2 * r[o + (t >= 2 ? t - 2 : 0)];
                r[o + t] = v - T.cp1 * r[o + t - 1];
            }
        } else {
            const double *tab = outer(q);
#pragma unroll
            for (int t = 1; t < S; t++) {
                double v = r[o + t];
                if (t >= 2) v = v - tab[t * kPenRow + 1] * r[o + (t >= 2 ? t - 2 : 0)];
                r[o + t] = v - tab[t * kPenRow] * r[o + t - 1];
            }
        }
        f1[m] = r[o + S - 1];
        f2[m] = r[o + S - 2];
    }
    double *cur = cb.a, *nxt = cb.b;
    auto scan = [&](const double *tabs, auto fwd, auto first) {
        constexpr bool FWD = decltype(fwd)::value;
#pragma unroll
        for (int m = 0; m < M; m++) {
            cur[(s0 + m) * L + lane] = f1[m];
            cur[PL + (s0 + m) * L + lane] = f2[m];
        }
        __syncthreads();
        if constexpr (decltype(first)::value) { if (threadIdx.x == 0) mid(); }
        for (int k = 0, d = 1; d < P; k++, d <<= 1) {
#pragma unroll
            for (int m = 0; m < M; m++) {
                const int q = s0 + m, at = q * L + lane;
                if (FWD ? q >= d : q + d < P) {
                    const double *mt = tabs + ((size_t)k * kMaxSeg + q) * 4;
                    const int o = at + (FWD ? -d : d) * L;
                    const double o1 = cur[o], o2 = cur[PL + o];
                    f1[m] = fma(__ldg(mt + 0), o1, fma(__ldg(mt + 1), o2, f1[m]));
                    f2[m] = fma(__ldg(mt + 2), o1, fma(__ldg(mt + 3), o2, f2[m]));
                }
                nxt[at] = f1[m];
                nxt[PL + at] = f2[m];
            }
            __syncthreads();
            double *t = cur; cur = nxt; nxt = t;
        }
    };
    scan(T.sf, std::true_type(), std::true_type());
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        const double c1 = q > 0 ? cur[(q - 1) * L + lane] : 0.0, c2 = q > 0 ? cur[PL + (q - 1) * L + lane] : 0.0;
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = fma(T.cg1[t], c1, fma(T.cg2[t], c2, r[o + t]));
#pragma unroll
            for (int t = S - 1; t >= 0; t--) {
                double v = r[o + t];
                if (t + 1 < S) v = v - T.cq1 * r[o + (t + 1 < S ? t + 1 : t)];
                if (t + 2 < S) v = v - T.cq2 * r[o + (t + 2 < S ? t + 2 : t)];
                r[o + t] = v * T.cid;
            }
        } else {
            const double *tab = outer(q);
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = fma(tab[t * kPenRow + 2], c1, fma(tab[t * kPenRow + 3], c2, r[o + t]));
#pragma unroll
            for (int t = S - 1; t >= 0; t--) {
                double v = r[o + t];
                if (t + 1 < S) v = v - tab[t * kPenRow + 5] * r[o + (t + 1 < S ? t + 1 : t)];
                if (t + 2 < S) v = v - tab[t * kPenRow + 6] * r[o + (t + 2 < S ? t + 2 : t)];
                r[o + t] = v * tab[t * kPenRow + 4];
            }
        }
        f1[m] = r[o];
        f2[m] = r[o + 1];
    }
    // the first values of the backward scan go to the buffer that nobody reads
    { double *t = cur; cur = nxt; nxt = t; }
    scan(T.sb, std::false_type(), std::false_type());
#pragma unroll
    for (int m = 0; m < M; m++) {
        const int q = s0 + m, o = m * S;
        const double e1 = q + 1 < P ? cur[(q + 1) * L + lane] : 0.0, e2 = q + 1 < P ? cur[PL + (q + 1) * L + lane] : 0.0;
        if (q >= T.slo && q < T.shi) {
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = fma(T.ch1[t], e1, fma(T.ch2[t], e2, r[o + t]));
        } else {
            const double *tab = outer(q);
#pragma unroll
            for (int t = 0; t < S; t++) r[o + t] = fma(tab[t * kPenRow + 7], e1, fma(tab[t * kPenRow + 8], e2, r[o + t]));
        }
    }
}

// ---- explicit right-hand sides ------------------------------------------
// v holds rows a-H .. a+S+H-1 on entry; the RHS of row a+t is written into
// v[t] (in place, ascending t: row a+t only needs v[t..t+2H]).  Rows follow
// the reference formulas term by term (Fortran evaluates left to right; the
// library is compiled without contraction).  Boundary rows belong to the
// first and last segment only: those read the few rows they need again
// through F (F(i): the operand at row i).

// DFDX_sym/_asym RHS, src/derivCDopt6_sym_tri.f:458-514,
// src/derivCDopt6_asym_tri.f:461-516  (H = 2).  Periodic DFDX,
// src/derivCDopt6_periodic.f:205-248: the interior formula on every row with
// wrapped halos (its f(i+-3) weight c1 is zero for the FDL3DI set).
template <int S, bool CYC, class RD, class V>
__device__ __forceinline__ void rhs_d1(V (&v)[S + 4], int a, int n, int asym, double fac, const Consts &K, const RD &F) {
#pragma unroll
    for (int t = 0; t < S; t++) {
        auto f = [&](int k) { return v[t + k + 2]; };
        v[t] = fac * (K.b1 * (f(2) - f(-2)) + K.a1 * (f(1) - f(-1)));
    }
    if (!CYC && a == 0) {
        const V f0 = F(0), f1 = F(1), f2 = F(2), f3 = F(3);
        v[0] = asym ? fac * (K.b1 * (f2 + f2) + K.a1 * (f1 + f1)) : V(0.0);
        v[1] = asym ? fac * (K.b1 * (f3 + f1) + K.a1 * (f2 - f0)) : fac * (K.b1 * (f3 - f1) + K.a1 * (f2 - f0));
    }
    if (!CYC && a + S == n) {
        const V f1 = F(n - 1), f0 = F(n - 2), m1 = F(n - 3), m2 = F(n - 4);
        v[S - 2] = fac * (K.closure1 * f1 + 5.0e-1 * f0 - m1 - K.closure2 * m2);
        v[S - 1] = fac * (2.5 * f1 - 2.0 * f0 - 5.0e-1 * m1);
    }
}

// D2FDX2_sym/_asym RHS, src/derivCDopt6_sym_tri.f:587-645,
// src/derivCDopt6_asym_tri.f:588-643  (H = 2).  Periodic D2FDX2,
// src/derivCDopt6_periodic.f:316-370, with zero f(i+-3) weight and centre
// weight 2(a2+b2).
template <int S, bool CYC, class RD, class V>
__device__ __forceinline__ void rhs_d2(V (&v)[S + 4], int a, int n, int asym, double fac, const Consts &K, const RD &F) {
#pragma unroll
    for (int t = 0; t < S; t++) {
        auto f = [&](int k) { return v[t + k + 2]; };
        v[t] = fac * (K.b2 * (f(2) + f(-2)) + K.a2 * (f(1) + f(-1)) - K.c2 * f(0));
    }
    if (!CYC && a == 0) {
        const V f0 = F(0), f1 = F(1), f2 = F(2), f3 = F(3);
        v[0] = asym ? V(0.0) : fac * (K.b2 * 2.0 * (f2 - f0) + K.a2 * 2.0 * (f1 - f0));
        v[1] = asym ? fac * (K.b2 * (f3 - 3.0 * f1) + K.a2 * (f2 - 2.0 * f1))
                    : fac * (K.b2 * (f3 - 2.0 * f1 + f1) + K.a2 * (f2 - 2.0 * f1 + f0));
    }
    if (!CYC && a + S == n) {
        const V f1 = F(n - 1), f0 = F(n - 2), m1 = F(n - 3), m2 = F(n - 4), m3 = F(n - 5);
        v[S - 2] = fac * (1.2375 * f1 - 3.0 * f0 + 2.325 * m1 - 6.0e-1 * m2 + 3.75e-2 * m3);
        v[S - 1] = fac * (1.3e1 * f1 - 2.7e1 * f0 + 1.5e1 * m1 - m2);
    }
}

// Compact_Filter_X_sym/_asym RHS, src/filters_sym.f:483-616,
// src/filters_asym.f:435-565  (H = 4).  Periodic Compact_Filter_X,
// src/filters_periodic.f:155-229: interior formula, wrapped halos.
template <int S, bool CYC, class RD>
__device__ __forceinline__ void rhs_filter(double (&v)[S + 8], int a, int n, int asym, const Consts &K, const RD &F) {
#pragma unroll
    for (int t = 0; t < S; t++) {
        auto f = [&](int k) { return v[t + k + 4]; };
        v[t] = K.fa4 * (f(4) + f(-4)) + K.fa3 * (f(3) + f(-3)) + K.fa2 * (f(2) + f(-2)) +
               K.fa1 * (f(1) + f(-1)) + K.fa0 * f(0);
    }
    if (!CYC && a == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            // rows outside the line: the mirrored row, with the sign of the symmetry
            auto pm = [&](int k) { return (asym && i - k < 0) ? F(i + k) - F(k - i) : F(i + k) + F(i - k < 0 ? k - i : i - k); };
            v[i] = (asym && i == 0) ? 0.0
                                    : K.fa4 * pm(4) + K.fa3 * pm(3) + K.fa2 * pm(2) + K.fa1 * pm(1) + K.fa0 * F(i);
        }
    }
    if (!CYC && a + S == n) {
        const double f0 = F(n - 1), f1 = F(n - 2), f2 = F(n - 3), f3 = F(n - 4), f4 = F(n - 5), f5 = F(n - 6), f6 = F(n - 7);
        v[S - 1] = K.bc1[1] * f0 + K.bc1[2] * f1 + K.bc1[3] * f2 + K.bc1[4] * f3 + K.bc1[5] * f4;
        v[S - 2] = K.bc2[1] * f0 + K.bc2[2] * f1 + K.bc2[3] * f2 + K.bc2[4] * f3 + K.bc2[5] * f4;
        v[S - 3] = K.bc3[2] * f4 + K.bc3[1] * f3 + K.bc3[0] * f2 + K.bc3[1] * f1 + K.bc3[2] * f0;
        v[S - 4] = K.bc4[3] * f6 + K.bc4[2] * f5 + K.bc4[1] * f4 + K.bc4[0] * f3 + K.bc4[1] * f2 + K.bc4[2] * f1 + K.bc4[3] * f0;
    }
}

// Gaussian_Filter_X, src/filters_sym.f:1119-1212: explicit, symmetric low end,
// last four points copied  (H = 4).  Periodic family,
// src/filters_periodic.f:601-675: interior formula, wrapped halos.
template <int S, bool CYC, class RD, class V>
__device__ __forceinline__ void rhs_gauss(V (&v)[S + 8], int a, int n, const Consts &K, const RD &F) {
    const double *g = K.ga;
#pragma unroll
    for (int t = 0; t < S; t++) {
        auto f = [&](int k) { return v[t + k + 4]; };
        v[t] = g[4] * (f(4) + f(-4)) + g[3] * (f(3) + f(-3)) + g[2] * (f(2) + f(-2)) + g[1] * (f(1) + f(-1)) +
               g[0] * f(0);
    }
    if (!CYC && a == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            auto pm = [&](int k) { return F(i + k) + F(i - k < 0 ? k - i : i - k); };
            v[i] = g[4] * pm(4) + g[3] * pm(3) + g[2] * pm(2) + g[1] * pm(1) + g[0] * F(i);
        }
    }
    if (!CYC && a + S == n) {
#pragma unroll
        for (int i = 0; i < 4; i++) v[S - 4 + i] = F(n - 4 + i);
    }
}

}  // namespace st
