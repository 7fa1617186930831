// st_solvers.cu - the general (per-line coefficient) tri- and pentadiagonal
// solvers: tridiagonal_serial / tridiagonal_periodic_serial
// (src/tridiagonal.f90:197-287) and pentadiagonal_serial /
// pentadiagonal_periodic_serial (src/pentadiagonal.f90:319-504).
// Arrays (lot,n) with lot fastest; the coefficients are read only (the
// reference works on copies of them), what the eliminations change goes to
// workspace fields, the right-hand side is solved in place.
//
// One thread per line, in blocks of one warp so that few lines still spread
// over all SMs, each step's arithmetic and order the reference's.  The chain
// of a line is a division and the products that depend on it per row; what a
// thread must not do besides is wait for its rows, so every sweep fetches the
// next U rows (4 to 8) into registers while it works on the U before them.
// Measured, 384 rows x 16384 lines, tridiagonal / periodic / pentadiagonal /
// periodic: 325 / 528 / 415 / 588 us.  At 2048 lines, 64 warps on the chip, it is
// 199 / 296 / 288 / 438 us: 260 ns, about 490 cycles, per row step of the
// first, which the chain's latency does not explain alone.  Row by row in
// blocks of 128 lines, with a copy of every array and an allocation per call,
// the four took 20.7 to 29.8 ms, as the allocations went.
#include <cfloat>
#include "st_internal.h"

namespace st {

namespace {

constexpr double kTinyPivot = (double)FLT_MIN;

// A sweep over rows i0, i0+dir, ... (cnt of them) of line L: get(row, d) loads
// the NF values of a row, step(row, d) works on them.
template <int U, int NF, class Get, class Step>
__device__ __forceinline__ void sweep(int i0, int dir, int cnt, Get get, Step step) {
    double x[U][NF], y[U][NF];
    auto fetch = [&](double (&d)[U][NF], int k0) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k0 + u < cnt) get(i0 + dir * (k0 + u), d[u]);
    };
    auto work = [&](double (&d)[U][NF], int k0) {
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k0 + u < cnt) step(i0 + dir * (k0 + u), d[u]);
    };
    fetch(x, 0);
    for (int k = 0; k < cnt; k += 2 * U) {
        fetch(y, k + U);
        work(x, k);
        fetch(x, k + 2 * U);
        work(y, k + U);
    }
}

__global__ void __launch_bounds__(32) k_tri(const double *__restrict__ A, const double *__restrict__ B,
                                            const double *__restrict__ C, double *__restrict__ R, double *__restrict__ bw,
                                            int n, int lot) {
    const int L = blockIdx.x * 32 + threadIdx.x;
    if (L >= lot) return;
    auto at = [&](int i) { return (size_t)i * lot + L; };
    double b = B[L], c = C[L], r = R[L];
    bw[L] = b;
    sweep<8, 4>(1, 1, n - 1,
                [&](int i, double (&d)[4]) { const size_t q = at(i); d[0] = A[q]; d[1] = B[q]; d[2] = C[q]; d[3] = R[q]; },
                [&](int i, double (&d)[4]) {
                    const double cs = d[0] / (b + kTinyPivot);
                    b = d[1] - c * cs;
                    r = d[3] - r * cs;
                    c = d[2];
                    bw[at(i)] = b;
                    R[at(i)] = r;
                });
    r = r / b;
    R[at(n - 1)] = r;
    sweep<8, 3>(n - 2, -1, n - 1, [&](int i, double (&d)[3]) { const size_t q = at(i); d[0] = C[q]; d[1] = bw[q]; d[2] = R[q]; },
                [&](int i, double (&d)[3]) {
                    r = (d[2] - d[0] * r) / (d[1] + kTinyPivot);
                    R[at(i)] = r;
                });
}

__global__ void __launch_bounds__(32) k_tri_per(const double *__restrict__ A, const double *__restrict__ B,
                                                const double *__restrict__ C, double *__restrict__ R, double *__restrict__ aw,
                                                double *__restrict__ bw, int n, int lot) {
    const int L = blockIdx.x * 32 + threadIdx.x;
    if (L >= lot) return;
    auto at = [&](int i) { return (size_t)i * lot + L; };
    double a = A[L], b = B[L], c = C[L], r = R[L];
    if (n == 1) { R[L] = r / (a + b + c); return; }
    if (n == 2) {
        const double c0 = c + a, a1 = A[at(1)] + C[at(1)], cs = a1 / b;
        const double b1 = B[at(1)] - c0 * cs;
        const double r1 = (R[at(1)] - r * cs) / b1;
        R[at(1)] = r1;
        R[L] = (r - c0 * r1) / b;
        return;
    }
    aw[L] = a;
    bw[L] = b;
    double bn = 0.0;                        // A(n-1) after the elimination
    sweep<6, 4>(1, 1, n - 1,
                [&](int i, double (&d)[4]) { const size_t q = at(i); d[0] = A[q]; d[1] = B[q]; d[2] = C[q]; d[3] = R[q]; },
                [&](int i, double (&d)[4]) {
                    const double cs = d[0] / b;
                    r = d[3] - r * cs;
                    R[at(i)] = r;
                    if (i == n - 1) { bn = d[1] - a * cs; return; }
                    b = d[1] - c * cs;
                    a = i == n - 2 ? d[2] - a * cs : -a * cs;
                    c = d[2];
                    bw[at(i)] = b;
                    aw[at(i)] = a;
                });
    // rows n-3 .. 0 with the row behind them (row n-2: a, b, and its r)
    double rn = r;
    r = R[at(n - 2)];
    sweep<6, 4>(n - 3, -1, n - 2,
                [&](int i, double (&d)[4]) { const size_t q = at(i); d[0] = C[q]; d[1] = bw[q]; d[2] = R[q]; d[3] = aw[q]; },
                [&](int i, double (&d)[4]) {
                    const double cs = d[0] / b;
                    r = d[2] - r * cs;
                    a = d[3] - a * cs;
                    b = d[1];
                    R[at(i)] = r;
                    aw[at(i)] = a;
                });
    const double cs = C[at(n - 1)] / b;
    rn = (rn - r * cs) / (bn - a * cs);
    R[at(n - 1)] = rn;
    sweep<8, 3>(n - 2, -1, n - 1, [&](int i, double (&d)[3]) { const size_t q = at(i); d[0] = R[q]; d[1] = aw[q]; d[2] = bw[q]; },
                [&](int i, double (&d)[3]) { R[at(i)] = (d[0] - d[1] * rn) / d[2]; });
}

__global__ void __launch_bounds__(32) k_pen(const double *__restrict__ A, const double *__restrict__ B, const double *__restrict__ C,
                                            const double *__restrict__ D, const double *__restrict__ E, double *__restrict__ R,
                                            double *__restrict__ cw, double *__restrict__ dw, int n, int lot) {
    const int L = blockIdx.x * 32 + threadIdx.x;
    if (L >= lot) return;
    auto at = [&](int i) { return (size_t)i * lot + L; };
    double c1 = C[L], d1 = D[L], e1 = E[L], r1 = R[L];            // row before
    if (n == 1) { R[L] = r1 / c1; return; }
    if (n == 2) {
        const double cs = B[at(1)] / c1, cc = C[at(1)] - d1 * cs, rr = (R[at(1)] - r1 * cs) / cc;
        R[at(1)] = rr;
        R[L] = (r1 - d1 * rr) / c1;
        return;
    }
    double c2 = 0.0, d2 = 0.0, e2 = 0.0, r2 = 0.0;                // the one before it
    cw[L] = c1;
    dw[L] = d1;
    sweep<4, 6>(1, 1, n - 1,
                [&](int i, double (&d)[6]) { const size_t q = at(i); d[0] = A[q]; d[1] = B[q]; d[2] = C[q]; d[3] = D[q]; d[4] = E[q]; d[5] = R[q]; },
                [&](int i, double (&d)[6]) {
                    double b = d[1], c = d[2], dd = d[3], r = d[5];
                    if (i >= 2) {
                        const double cs = d[0] / (c2 + kTinyPivot);
                        b = b - d2 * cs;
                        c = c - e2 * cs;
                        r = r - r2 * cs;
                    }
                    const double cs = b / (c1 + kTinyPivot);
                    c = c - d1 * cs;
                    dd = dd - e1 * cs;
                    r = r - r1 * cs;
                    c2 = c1; d2 = d1; e2 = e1; r2 = r1;
                    c1 = c; d1 = dd; e1 = d[4]; r1 = r;
                    cw[at(i)] = c;
                    dw[at(i)] = dd;
                    R[at(i)] = r;
                });
    r1 = r1 / (c1 + kTinyPivot);                                  // row n-1
    R[at(n - 1)] = r1;
    r2 = (r2 - d2 * r1) / (c2 + kTinyPivot);                      // row n-2
    R[at(n - 2)] = r2;
    sweep<6, 4>(n - 3, -1, n - 2,
                [&](int i, double (&d)[4]) { const size_t q = at(i); d[0] = cw[q]; d[1] = dw[q]; d[2] = E[q]; d[3] = R[q]; },
                [&](int i, double (&d)[4]) {
                    const double r = (d[3] - d[1] * r2 - d[2] * r1) / (d[0] + kTinyPivot);
                    r1 = r2;
                    r2 = r;
                    R[at(i)] = r;
                });
}

// n >= 5
__global__ void __launch_bounds__(32) k_pen_per(const double *__restrict__ A, const double *__restrict__ B,
                                                const double *__restrict__ C, const double *__restrict__ D,
                                                const double *__restrict__ E, double *__restrict__ R, double *__restrict__ cw,
                                                double *__restrict__ dw, double *__restrict__ s1, double *__restrict__ s2, int n,
                                                int lot) {
    const int L = blockIdx.x * 32 + threadIdx.x;
    if (L >= lot) return;
    auto at = [&](int i) { return (size_t)i * lot + L; };
    // a row's right-hand side and its columns n-2 and n-1 (p, q)
    struct Row { double c, d, e, r, p, q; };
    Row x1{0, 0, 0, 0, 0, 0}, x2{0, 0, 0, 0, 0, 0};               // the row before, the one before it
    Row lo0{}, lo1{};                                             // rows n-2 and n-1 after the sweep
    sweep<4, 6>(0, 1, n,
                [&](int i, double (&d)[6]) { const size_t q = at(i); d[0] = A[q]; d[1] = B[q]; d[2] = C[q]; d[3] = D[q]; d[4] = E[q]; d[5] = R[q]; },
                [&](int i, double (&d)[6]) {
                    double b = d[1];
                    Row x{d[2], d[3], d[4], d[5], 0.0, 0.0};
                    if (i == 0) x.p = d[0];
                    if (i == n - 4) x.p = x.p + d[4];
                    if (i == n - 3) x.p = d[3];
                    if (i == n - 2) x.p = d[2];
                    if (i == n - 1) x.p = d[1];
                    if (i == 0) x.q = d[1];
                    if (i == 1) x.q = d[0];
                    if (i == n - 3) x.q = x.q + d[4];
                    if (i == n - 2) x.q = d[3];
                    if (i == n - 1) x.q = d[2];
                    if (i >= 2) {
                        const double cs = d[0] / x2.c;
                        b = b - x2.d * cs;
                        x.c = x.c - x2.e * cs;
                        x.r = x.r - x2.r * cs;
                        x.p = x.p - x2.p * cs;
                        x.q = x.q - x2.q * cs;
                    }
                    if (i >= 1 && i <= n - 2) {
                        const double cs = b / x1.c;
                        x.c = x.c - x1.d * cs;
                        x.d = x.d - x1.e * cs;
                        x.r = x.r - x1.r * cs;
                        x.p = x.p - x1.p * cs;
                        x.q = x.q - x1.q * cs;
                    }
                    x2 = x1;
                    x1 = x;
                    if (i == n - 2) lo0 = x;
                    if (i == n - 1) { lo1 = x; return; }
                    const size_t w = at(i);
                    cw[w] = x.c; dw[w] = x.d; s1[w] = x.p; s2[w] = x.q; R[w] = x.r;
                });
    // rows n-4 .. 0 with the two behind them (from row n-3 up)
    {
        const size_t w = at(n - 3);
        x1 = Row{cw[w], 0.0, 0.0, R[w], s1[w], s2[w]};
        x2 = x1;
    }
    sweep<4, 6>(n - 4, -1, n - 3,
                [&](int i, double (&d)[6]) { const size_t w = at(i); d[0] = cw[w]; d[1] = dw[w]; d[2] = E[w]; d[3] = R[w]; d[4] = s1[w]; d[5] = s2[w]; },
                [&](int i, double (&d)[6]) {
                    Row x{d[0], d[1], d[2], d[3], d[4], d[5]};
                    if (i <= n - 5) {
                        const double cs = x.e / x2.c;
                        x.r = x.r - x2.r * cs;
                        x.p = x.p - x2.p * cs;
                        x.q = x.q - x2.q * cs;
                    }
                    const double cs = x.d / x1.c;
                    x.r = x.r - x1.r * cs;
                    x.p = x.p - x1.p * cs;
                    x.q = x.q - x1.q * cs;
                    x2 = x1;
                    x1 = x;
                    const size_t w = at(i);
                    R[w] = x.r; s1[w] = x.p; s2[w] = x.q;
                });
    // x1, x2: rows 0 and 1
    double cs = lo0.e / x1.c;
    lo0.r = lo0.r - x1.r * cs;
    lo0.p = lo0.p - x1.p * cs;
    lo0.q = lo0.q - x1.q * cs;
    cs = lo1.d / x1.c;
    lo1.r = lo1.r - x1.r * cs;
    lo1.p = lo1.p - x1.p * cs;
    lo1.q = lo1.q - x1.q * cs;
    cs = lo1.e / x2.c;
    lo1.r = lo1.r - x2.r * cs;
    lo1.p = lo1.p - x2.p * cs;
    lo1.q = lo1.q - x2.q * cs;
    cs = lo1.p / lo0.p;
    lo1.r = lo1.r - lo0.r * cs;
    lo1.q = lo1.q - lo0.q * cs;
    const double rn = lo1.r / lo1.q, rm = (lo0.r - lo0.q * rn) / lo0.p;
    R[at(n - 1)] = rn;
    R[at(n - 2)] = rm;
    sweep<6, 4>(n - 3, -1, n - 2, [&](int i, double (&d)[4]) { const size_t w = at(i); d[0] = R[w]; d[1] = s1[w]; d[2] = s2[w]; d[3] = cw[w]; },
                [&](int i, double (&d)[4]) { R[at(i)] = (d[0] - d[1] * rm - d[2] * rn) / d[3]; });
}

}  // namespace

// The solvers' workspace: grows to the largest call's need; one above kKeep is
// given back when its call ends, any when a scratch field finds no room.
constexpr size_t kKeep = (size_t)1 << 30;
void solver_workspace_free(st_ctx *c) {
    if (c->solver_ws) { cudaStreamSynchronize(c->stream); cudaFree(c->solver_ws); }
    cudaGetLastError();
    c->solver_ws = nullptr;
    c->solver_ws_bytes = 0;
}
double *solver_workspace(st_ctx *c, size_t bytes) {
    if (bytes > c->solver_ws_bytes) {
        solver_workspace_free(c);
        if (cudaMalloc(&c->solver_ws, bytes) != cudaSuccess) { cudaGetLastError(); c->solver_ws = nullptr; return nullptr; }
        c->solver_ws_bytes = bytes;
    }
    return (double *)c->solver_ws;
}
void solver_workspace_trim(st_ctx *c) {
    if (c->solver_ws_bytes > kKeep) solver_workspace_free(c);
}

// fields of workspace the solvers need beside their arguments
int solver_fields(bool pen, int nper) { return pen ? (nper ? 4 : 2) : (nper ? 2 : 1); }

int dev_tridiagonal(st_ctx *c, const double *A, const double *B, const double *C, double *R, double *ws, int n, int lot,
                    int nper) {
    const size_t N = (size_t)n * lot;
    const int blocks = (lot + 31) / 32;
    const int pi = prof_start(c, "k_tri_general", 40.0 * N);
    if (nper == 0) k_tri<<<blocks, 32, 0, c->stream>>>(A, B, C, R, ws, n, lot);
    else k_tri_per<<<blocks, 32, 0, c->stream>>>(A, B, C, R, ws, ws + N, n, lot);
    prof_stop(c, pi);
    ST_CUDA(c, cudaGetLastError());
    return ST_OK;
}

int dev_pentadiagonal(st_ctx *c, const double *A, const double *B, const double *C, const double *D, const double *E, double *R,
                      double *ws, int n, int lot, int nper) {
    if (nper && n < 5) return fail(c, ST_E_UNSUPPORTED, "periodic pentadiagonal needs n >= 5");
    const size_t N = (size_t)n * lot;
    const int blocks = (lot + 31) / 32;
    const int pi = prof_start(c, "k_pen_general", 56.0 * N);
    if (nper == 0) k_pen<<<blocks, 32, 0, c->stream>>>(A, B, C, D, E, R, ws, ws + N, n, lot);
    else k_pen_per<<<blocks, 32, 0, c->stream>>>(A, B, C, D, E, R, ws, ws + N, ws + 2 * N, ws + 3 * N, n, lot);
    prof_stop(c, pi);
    ST_CUDA(c, cudaGetLastError());
    return ST_OK;
}

}  // namespace st
