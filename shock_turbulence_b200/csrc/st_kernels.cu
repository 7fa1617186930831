// st_kernels.cu - compact derivative, compact filter and Gaussian filter line
// operators (bounded-line instantiations and the entry points of both
// families), and the general (per-line coefficient) tri/pentadiagonal solvers.
#include <initializer_list>
#include "st_linekern.cuh"

namespace st {

int launch_rec(st_ctx *c, RecId id, LineArgs &a, const double *const *in, double *const *out) {
    return launch_rec_t<false, double>(c, id, a, in, out);
}

// the context's family and the field type pick the instantiation
static int launch(st_ctx *c, RecId id, LineArgs &a, const double *const *in, double *const *out) {
    return c->p.family == ST_FAMILY_PERIODIC ? launch_rec_cyc(c, id, a, in, out) : launch_rec(c, id, a, in, out);
}
static int launch(st_ctx *c, RecId id, LineArgsF &a, const float *const *in, float *const *out) {
    return c->p.family == ST_FAMILY_PERIODIC ? launch_rec_cyc_f32(c, id, a, in, out) : launch_rec_f32(c, id, a, in, out);
}

// cuTensorMapEncodeTiled through the runtime (the library does not link libcuda)
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (EncodeTiled)f;
    }();
    return fn;
}

// Encoded anew for every launch (0.05 us on the host); L2 promotion to 256
// bytes: neighbouring CTAs read the other half (2 % on x and z lines).
int line_map(st_ctx *c, CUtensorMap *m, const void *p, bool f32, int dir, int nl, int box) {
    const EncodeTiled enc = encode_tiled();
    if (!enc) return fail(c, ST_E_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t es = f32 ? 4 : 8, my = c->dm.n[1], mz = c->dm.n[2], mx = c->dm.n[0], na = (cuuint64_t)c->na;
    cuuint64_t dims[4] = {my, mz, mx, na}, str[3] = {my * es, my * mz * es, (cuuint64_t)c->dm.n3 * es};
    cuuint32_t b[4] = {(cuuint32_t)nl, dir == 0 ? 1u : (cuuint32_t)box, dir == 0 ? (cuuint32_t)box : 1u, 1u};
    if (dir == 1) {   // the lines of all cases follow one another
        const cuuint64_t rc = 128 / es, ch = my / rc;
        dims[0] = rc; dims[1] = mz * mx * na; dims[2] = ch; dims[3] = 1;
        str[1] = 128; str[2] = my * es * dims[1];
        b[0] = (cuuint32_t)rc; b[1] = (cuuint32_t)nl; b[2] = (cuuint32_t)ch;
    }
    const cuuint32_t one[4] = {1, 1, 1, 1};
    const CUresult r = enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void *>(p),
                           dims, str, b, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           dir == 1 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(c, ST_E_CUDA, "cuTensorMapEncodeTiled failed (field not 16-byte aligned?)");
    return ST_OK;
}

template <class T>
static LineArgsT<T> make_args(st_ctx *c, int dir) {
    LineArgsT<T> a{};
    a.dir = dir;
    a.n = c->dm.n[dir];
    a.c = c->k;
    return a;
}
template <class T>
static const TriTabT<T> &tri_tab(st_ctx *c, int dir, int kind) {
    if constexpr (sizeof(T) == 8) return c->tri[dir][kind];
    else return c->trif[dir][kind];
}
// bulk copies and tensor maps need 16-byte aligned fields
static int aligned(st_ctx *c, const void *p) {
    if (reinterpret_cast<uintptr_t>(p) & 15) return fail(c, ST_E_ARG, "line operators need 16-byte aligned fields");
    return ST_OK;
}

// first-derivative arguments of operation k of a launch (its output, sign of
// the symmetry, accumulation and factor), src/derivCDopt6_sym_tri.f:424
template <class T>
static void set_d1(st_ctx *c, LineArgsT<T> &a, int k, int asym, int iadd, double cadd) {
    a.op[k].asym = asym;
    a.op[k].fac1 = cadd * c->s1[a.dir] * (double)(a.n - 1);
    a.op[k].t1 = tri_tab<T>(c, a.dir, asym ? K_D1A : K_D1S);
    a.red[k] = iadd;
}

template <class T>
static int dfd_t(st_ctx *c, int dir, int asym, const ProdT<T> &F, T *dF, int iadd, double cadd) {
    static const RecId rec[] = {R_D1, R_MUL, R_ADDMUL, R_MULMUL, R_SPEC, R_SPECT, R_HMULADD};
    static const int nin[] = {1, 2, 3, 3, 3, 4, 3};
    LineArgsT<T> a = make_args<T>(c, dir);
    set_d1(c, a, 0, asym, iadd, cadd);
    a.k0 = F.k0; a.k1 = F.k1; a.k2 = F.k2;
    // a*b/2 + c in the FP32 mode: the derivative of a*b with half the factor,
    // plus that of c
    if (F.op == PR_HMULADD && sizeof(T) == 4) { a.op[1] = a.op[0]; a.op[1].fac1 = 0.5 * a.op[0].fac1; }
    const T *in[4] = {F.a, F.b, F.c, F.d};
    for (int k = 0; k < nin[F.op]; k++) ST_TRY(aligned(c, in[k]));
    ST_TRY(aligned(c, dF));
    return launch(c, rec[F.op], a, in, &dF);
}

// D2F*2: d2F, and dF where given (iadd)
template <class T>
static int d2_t(st_ctx *c, int dir, int asym, const T *F, T *dF, T *d2F, int iadd, int red) {
    LineArgsT<T> a = make_args<T>(c, dir);
    a.op[0].asym = asym;
    a.op[0].fac2 = ((double)((a.n - 1) * (a.n - 1))) * c->s2[dir];   // src/derivCDopt6_sym_tri.f:554
    a.op[0].t2 = tri_tab<T>(c, dir, asym ? K_D2A : K_D2S);
    a.red[0] = red;
    ST_TRY(aligned(c, F)); ST_TRY(aligned(c, d2F));
    if (iadd) { ST_TRY(aligned(c, dF)); set_d1(c, a, 1, asym, 0, 1.0); }
    T *out[2] = {d2F, dF};
    return launch(c, iadd ? R_D2D1 : R_D2, a, &F, out);
}

template <class T>
static int lap_t(st_ctx *c, int dir, const T *F, T *out, int iadd, bool second) {
    if (second) return d2_t<T>(c, dir, 0, F, (T *)nullptr, out, 0, iadd);
    LineArgsT<T> a = make_args<T>(c, dir);
    set_d1(c, a, 0, 0, iadd, 1.0);
    a.op[0].t2 = tri_tab<T>(c, dir, K_D1A);
    ST_TRY(aligned(c, F)); ST_TRY(aligned(c, out));
    return launch(c, R_LAP, a, &F, &out);
}

template <class T>
static int gauss_t(st_ctx *c, int dir, const T *F, T *Fg) {
    LineArgsT<T> a = make_args<T>(c, dir);
    ST_TRY(aligned(c, F)); ST_TRY(aligned(c, Fg));
    return launch(c, R_GAUSS, a, &F, &Fg);
}

static Prod plain(const double *F) { Prod p{}; p.op = PR_A; p.a = F; return p; }
static ProdF plain(const float *F) { ProdF p{}; p.op = PR_A; p.a = F; return p; }

int dev_dfd(st_ctx *c, int dir, int asym, const double *F, double *dF, int iadd, double cadd) {
    return dfd_t<double>(c, dir, asym, plain(F), dF, iadd, cadd);
}
int dev_dfd_prod(st_ctx *c, int dir, int asym, const Prod &F, double *dF, int iadd, double cadd) {
    return dfd_t<double>(c, dir, asym, F, dF, iadd, cadd);
}
int dev_d2fd2(st_ctx *c, int dir, int asym, const double *F, double *dF, double *d2F, int iadd) {
    return d2_t<double>(c, dir, asym, F, dF, d2F, iadd, 0);
}
int dev_lap(st_ctx *c, int dir, const double *F, double *out, int iadd, bool second) {
    return lap_t<double>(c, dir, F, out, iadd, second);
}
int dev_filter(st_ctx *c, int dir, int asym, const double *F, double *F0) {
    LineArgs a = make_args<double>(c, dir);
    a.op[0].asym = asym;
    a.p = c->pen[dir][asym ? K_FA : K_FS];
    ST_TRY(aligned(c, F)); ST_TRY(aligned(c, F0));
    return launch(c, R_FILTER, a, &F, &F0);
}
int dev_gauss(st_ctx *c, int dir, const double *F, double *Fg) { return gauss_t<double>(c, dir, F, Fg); }

// FP32 mode (float fields and arithmetic, two lines per thread)
int dev_dfd_f(st_ctx *c, int dir, int asym, const float *F, float *dF, int iadd, double cadd) {
    return dfd_t<float>(c, dir, asym, plain(F), dF, iadd, cadd);
}
int dev_dfd_prod_f(st_ctx *c, int dir, int asym, const ProdF &F, float *dF, int iadd, double cadd) {
    return dfd_t<float>(c, dir, asym, F, dF, iadd, cadd);
}
int dev_d2fd2_f(st_ctx *c, int dir, int asym, const float *F, float *dF, float *d2F, int iadd) {
    return d2_t<float>(c, dir, asym, F, dF, d2F, iadd, 0);
}
int dev_lap_f(st_ctx *c, int dir, const float *F, float *out, int iadd, bool second) {
    return lap_t<float>(c, dir, F, out, iadd, second);
}
int dev_gauss_f(st_ctx *c, int dir, const float *F, float *Fg) { return gauss_t<float>(c, dir, F, Fg); }

// ---- two first derivatives along one direction, one launch ---------------------
// The pairs that the RHS routines form share operand fields, so that one
// launch reads each field once:
//   A  F, U F            B  a b, c (a b)            C  the species flux, its energy counterpart
//   D  a u, (b + c) u    E  a u, b u
// Each operation is the single one's arithmetic, so the results are those of
// two launches.  Any other pair, and one whose operations add to the same
// field, runs as two launches.
template <class T>
static int dfd_pair_t(st_ctx *c, int dir, const D1SpecT<T> *ops) {
    const ProdT<T> &p = ops[0].F, &q = ops[1].F;
    LineArgsT<T> a = make_args<T>(c, dir);
    const T *in[4] = {nullptr, nullptr, nullptr, nullptr};
    int id = -1, ni = 0;
    auto use = [&](RecId r, std::initializer_list<const T *> f) { id = r; for (const T *x : f) in[ni++] = x; };
    if (ops[0].dF != ops[1].dF) {
        if (p.op == PR_A && q.op == PR_MUL && q.b == p.a) use(R_PAIRA, {p.a, q.a});
        else if (p.op == PR_MUL && q.op == PR_MULMUL && q.a == p.a && q.b == p.b) use(R_PAIRB, {p.a, p.b, q.c});
        else if (p.op == PR_SPEC && q.op == PR_SPECT && q.a == p.a && q.b == p.b && q.c == p.c &&
                 c->p.family != ST_FAMILY_PERIODIC)
            use(R_PAIRC, {p.a, p.b, p.c, q.d});
        else if (p.op == PR_MUL && q.op == PR_ADDMUL && q.c == p.b) use(R_PAIRD, {p.a, p.b, q.a, q.b});
        else if (p.op == PR_MUL && q.op == PR_MUL && q.b == p.b) use(R_PAIRE, {p.a, p.b, q.a});
    }
    if (id < 0) {
        for (int i = 0; i < 2; i++) ST_TRY(dfd_t<T>(c, dir, ops[i].asym, ops[i].F, ops[i].dF, ops[i].iadd, ops[i].cadd));
        return ST_OK;
    }
    T *out[2];
    for (int i = 0; i < 2; i++) {
        set_d1(c, a, i, ops[i].asym, ops[i].iadd, ops[i].cadd);
        out[i] = ops[i].dF;
        ST_TRY(aligned(c, out[i]));
    }
    for (int k = 0; k < ni; k++) ST_TRY(aligned(c, in[k]));
    a.k0 = q.k0; a.k1 = q.k1; a.k2 = q.k2;
    return launch(c, (RecId)id, a, in, out);
}

int dev_dfd_pair(st_ctx *c, int dir, const D1SpecT<double> *ops) { return dfd_pair_t(c, dir, ops); }
int dev_dfd_pair_f(st_ctx *c, int dir, const D1SpecT<float> *ops) { return dfd_pair_t(c, dir, ops); }

// ---- general solvers (per-line coefficients), thread per line ---------------
// tridiagonal_serial / tridiagonal_periodic_serial, src/tridiagonal.f90:197-287.
// Arrays (lot,n) with lot fastest; A,B,C are copied into scratch first (the
// reference's A=A1; B=B1; C=C1).
__global__ void k_tri_general(double *a, double *b, const double *cc, double *R, int n, int lot,
                              int nper) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= lot) return;
    const double tiny = (double)FLT_MIN;
#define A_(i) a[(size_t)(i) * lot + L]
#define B_(i) b[(size_t)(i) * lot + L]
#define C_(i) cc[(size_t)(i) * lot + L]
#define R_(i) R[(size_t)(i) * lot + L]
    if (nper == 0) {
        for (int i = 1; i < n; i++) {
            double cs = A_(i) / (B_(i - 1) + tiny);
            B_(i) = B_(i) - C_(i - 1) * cs;
            R_(i) = R_(i) - R_(i - 1) * cs;
        }
        R_(n - 1) = R_(n - 1) / B_(n - 1);
        for (int i = n - 2; i >= 0; i--) R_(i) = (R_(i) - C_(i) * R_(i + 1)) / (B_(i) + tiny);
        return;
    }
    double c0 = C_(0);
    if (n == 1) { R_(0) = R_(0) / (A_(0) + B_(0) + C_(0)); return; }
    if (n == 2) {
        c0 = C_(0) + A_(0);
        A_(1) = A_(1) + C_(1);
        double cs = A_(1) / B_(0);
        B_(1) = B_(1) - c0 * cs;
        R_(1) = R_(1) - R_(0) * cs;
        R_(1) = R_(1) / B_(1);
        R_(0) = (R_(0) - c0 * R_(1)) / B_(0);
        return;
    }
    for (int i = 1; i <= n - 3; i++) {
        double cs = A_(i) / B_(i - 1);
        B_(i) = B_(i) - C_(i - 1) * cs;
        R_(i) = R_(i) - R_(i - 1) * cs;
        A_(i) = -A_(i - 1) * cs;
    }
    int i = n - 2;
    double cs = A_(i) / B_(i - 1);
    B_(i) = B_(i) - C_(i - 1) * cs;
    R_(i) = R_(i) - R_(i - 1) * cs;
    A_(i) = C_(i) - A_(i - 1) * cs;
    i = n - 1;
    cs = A_(i) / B_(i - 1);
    R_(i) = R_(i) - R_(i - 1) * cs;
    A_(i) = B_(i) - A_(i - 1) * cs;
    for (i = n - 3; i >= 0; i--) {
        cs = C_(i) / B_(i + 1);
        R_(i) = R_(i) - R_(i + 1) * cs;
        A_(i) = A_(i) - A_(i + 1) * cs;
    }
    cs = C_(n - 1) / B_(0);
    R_(n - 1) = R_(n - 1) - R_(0) * cs;
    A_(n - 1) = A_(n - 1) - A_(0) * cs;
    R_(n - 1) = R_(n - 1) / A_(n - 1);
    for (i = n - 2; i >= 0; i--) R_(i) = (R_(i) - A_(i) * R_(n - 1)) / B_(i);
#undef A_
#undef B_
#undef C_
#undef R_
}

// pentadiagonal_serial / pentadiagonal_periodic_serial,
// src/pentadiagonal.f90:319-504 (n >= 5 for the periodic path)
__global__ void k_pen_general(double *A, double *B, double *C, double *D, double *E, double *R,
                              double *s1, double *s2, int n, int lot, int nper) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= lot) return;
    const double tiny = (double)FLT_MIN;
#define X_(arr, i) arr[(size_t)(i) * lot + L]
    if (nper == 0) {
        if (n == 1) { X_(R, 0) = X_(R, 0) / X_(C, 0); return; }
        if (n == 2) {
            double cs = X_(B, 1) / X_(C, 0);
            X_(C, 1) = X_(C, 1) - X_(D, 0) * cs;
            X_(R, 1) = X_(R, 1) - X_(R, 0) * cs;
            X_(R, 1) = X_(R, 1) / X_(C, 1);
            X_(R, 0) = (X_(R, 0) - X_(D, 0) * X_(R, 1)) / X_(C, 0);
            return;
        }
        for (int i = 0; i <= n - 3; i++) {
            double cs = X_(B, i + 1) / (X_(C, i) + tiny);
            X_(C, i + 1) = X_(C, i + 1) - X_(D, i) * cs;
            X_(D, i + 1) = X_(D, i + 1) - X_(E, i) * cs;
            X_(R, i + 1) = X_(R, i + 1) - X_(R, i) * cs;
            cs = X_(A, i + 2) / (X_(C, i) + tiny);
            X_(B, i + 2) = X_(B, i + 2) - X_(D, i) * cs;
            X_(C, i + 2) = X_(C, i + 2) - X_(E, i) * cs;
            X_(R, i + 2) = X_(R, i + 2) - X_(R, i) * cs;
        }
        double cs = X_(B, n - 1) / (X_(C, n - 2) + tiny);
        X_(C, n - 1) = X_(C, n - 1) - X_(D, n - 2) * cs;
        X_(R, n - 1) = X_(R, n - 1) - X_(R, n - 2) * cs;
        X_(R, n - 1) = X_(R, n - 1) / (X_(C, n - 1) + tiny);
        X_(R, n - 2) = (X_(R, n - 2) - X_(D, n - 2) * X_(R, n - 1)) / (X_(C, n - 2) + tiny);
        for (int i = n - 3; i >= 0; i--)
            X_(R, i) = (X_(R, i) - X_(D, i) * X_(R, i + 1) - X_(E, i) * X_(R, i + 2)) / (X_(C, i) + tiny);
        return;
    }
    for (int i = 0; i < n; i++) { X_(s1, i) = 0.0; X_(s2, i) = 0.0; }
    if (n == 4) for (int i = 0; i < 4; i++) { X_(A, i) = X_(A, i) + X_(E, i); X_(E, i) = 0.0; }
    X_(s1, 0) = X_(A, 0);
    X_(s1, n - 4) = X_(s1, n - 4) + X_(E, n - 4);
    X_(s1, n - 3) = X_(D, n - 3);
    X_(s1, n - 2) = X_(C, n - 2);
    X_(s1, n - 1) = X_(B, n - 1);
    X_(s2, 0) = X_(B, 0);
    X_(s2, 1) = X_(A, 1);
    X_(s2, n - 3) = X_(s2, n - 3) + X_(E, n - 3);
    X_(s2, n - 2) = X_(D, n - 2);
    X_(s2, n - 1) = X_(C, n - 1);
    for (int i = 0; i <= n - 3; i++) {
        double cs = X_(B, i + 1) / X_(C, i);
        X_(C, i + 1) = X_(C, i + 1) - X_(D, i) * cs;
        X_(D, i + 1) = X_(D, i + 1) - X_(E, i) * cs;
        X_(R, i + 1) = X_(R, i + 1) - X_(R, i) * cs;
        X_(s1, i + 1) = X_(s1, i + 1) - X_(s1, i) * cs;
        X_(s2, i + 1) = X_(s2, i + 1) - X_(s2, i) * cs;
        cs = X_(A, i + 2) / X_(C, i);
        X_(B, i + 2) = X_(B, i + 2) - X_(D, i) * cs;
        X_(C, i + 2) = X_(C, i + 2) - X_(E, i) * cs;
        X_(R, i + 2) = X_(R, i + 2) - X_(R, i) * cs;
        X_(s1, i + 2) = X_(s1, i + 2) - X_(s1, i) * cs;
        X_(s2, i + 2) = X_(s2, i + 2) - X_(s2, i) * cs;
    }
    for (int i = n - 3; i >= 2; i--) {
        double cs = X_(D, i - 1) / X_(C, i);
        X_(R, i - 1) = X_(R, i - 1) - X_(R, i) * cs;
        X_(s1, i - 1) = X_(s1, i - 1) - X_(s1, i) * cs;
        X_(s2, i - 1) = X_(s2, i - 1) - X_(s2, i) * cs;
        cs = X_(E, i - 2) / X_(C, i);
        X_(R, i - 2) = X_(R, i - 2) - X_(R, i) * cs;
        X_(s1, i - 2) = X_(s1, i - 2) - X_(s1, i) * cs;
        X_(s2, i - 2) = X_(s2, i - 2) - X_(s2, i) * cs;
    }
    {
        double cs = X_(D, 0) / X_(C, 1);
        X_(R, 0) = X_(R, 0) - X_(R, 1) * cs;
        X_(s1, 0) = X_(s1, 0) - X_(s1, 1) * cs;
        X_(s2, 0) = X_(s2, 0) - X_(s2, 1) * cs;
    }
    double cs = X_(E, n - 2) / X_(C, 0);
    X_(R, n - 2) = X_(R, n - 2) - X_(R, 0) * cs;
    X_(s1, n - 2) = X_(s1, n - 2) - X_(s1, 0) * cs;
    X_(s2, n - 2) = X_(s2, n - 2) - X_(s2, 0) * cs;
    cs = X_(D, n - 1) / X_(C, 0);
    X_(R, n - 1) = X_(R, n - 1) - X_(R, 0) * cs;
    X_(s1, n - 1) = X_(s1, n - 1) - X_(s1, 0) * cs;
    X_(s2, n - 1) = X_(s2, n - 1) - X_(s2, 0) * cs;
    cs = X_(E, n - 1) / X_(C, 1);
    X_(R, n - 1) = X_(R, n - 1) - X_(R, 1) * cs;
    X_(s1, n - 1) = X_(s1, n - 1) - X_(s1, 1) * cs;
    X_(s2, n - 1) = X_(s2, n - 1) - X_(s2, 1) * cs;
    cs = X_(s1, n - 1) / X_(s1, n - 2);
    X_(R, n - 1) = X_(R, n - 1) - X_(R, n - 2) * cs;
    X_(s2, n - 1) = X_(s2, n - 1) - X_(s2, n - 2) * cs;
    X_(R, n - 1) = X_(R, n - 1) / X_(s2, n - 1);
    X_(R, n - 2) = (X_(R, n - 2) - X_(s2, n - 2) * X_(R, n - 1)) / X_(s1, n - 2);
    for (int i = n - 3; i >= 0; i--)
        X_(R, i) = (X_(R, i) - X_(s1, i) * X_(R, n - 2) - X_(s2, i) * X_(R, n - 1)) / X_(C, i);
#undef X_
}

int dev_tridiagonal(st_ctx *c, const double *A, const double *B, const double *C, double *R, int n,
                    int lot, int nper) {
    size_t N = (size_t)n * lot;
    double *a = nullptr, *b = nullptr;
    ST_CUDA(c, cudaMallocAsync(&a, 2 * N * sizeof(double), c->stream));
    b = a + N;
    ST_CUDA(c, cudaMemcpyAsync(a, A, N * 8, cudaMemcpyDeviceToDevice, c->stream));
    ST_CUDA(c, cudaMemcpyAsync(b, B, N * 8, cudaMemcpyDeviceToDevice, c->stream));
    int pi = prof_start(c, "k_tri_general", 32.0 * N);
    k_tri_general<<<(lot + 127) / 128, 128, 0, c->stream>>>(a, b, C, R, n, lot, nper);
    prof_stop(c, pi);
    cudaError_t e = cudaGetLastError();
    cudaFreeAsync(a, c->stream);
    if (e != cudaSuccess) return fail(c, ST_E_CUDA, cudaGetErrorString(e));
    return ST_OK;
}

int dev_pentadiagonal(st_ctx *c, const double *A, const double *B, const double *C, const double *D,
                      const double *E, double *R, int n, int lot, int nper) {
    if (nper && n < 5) return fail(c, ST_E_UNSUPPORTED, "periodic pentadiagonal needs n >= 5");
    size_t N = (size_t)n * lot;
    double *buf = nullptr;
    ST_CUDA(c, cudaMallocAsync(&buf, 7 * N * sizeof(double), c->stream));
    double *a = buf, *b = buf + N, *cc = buf + 2 * N, *d = buf + 3 * N, *e = buf + 4 * N;
    double *s1 = buf + 5 * N, *s2 = buf + 6 * N;
    const double *src[5] = {A, B, C, D, E};
    double *dst[5] = {a, b, cc, d, e};
    for (int q = 0; q < 5; q++)
        ST_CUDA(c, cudaMemcpyAsync(dst[q], src[q], N * 8, cudaMemcpyDeviceToDevice, c->stream));
    int pi = prof_start(c, "k_pen_general", 48.0 * N);
    k_pen_general<<<(lot + 127) / 128, 128, 0, c->stream>>>(a, b, cc, d, e, R, s1, s2, n, lot, nper);
    prof_stop(c, pi);
    cudaError_t er = cudaGetLastError();
    cudaFreeAsync(buf, c->stream);
    if (er != cudaSuccess) return fail(c, ST_E_CUDA, cudaGetErrorString(er));
    return ST_OK;
}

}  // namespace st
