// st_kernels.cu - compact derivative, compact filter and Gaussian filter line
// operators (bounded-line instantiations and the entry points of both
// families).
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
    RecId id;
    int nin;
    switch (F.op) {
        case PR_A: id = R_D1; nin = 1; break;
        case PR_MUL: id = R_MUL; nin = 2; break;
        case PR_ADDMUL: id = R_ADDMUL; nin = 3; break;
        case PR_MULPLUS: id = R_MULPLUS; nin = 3; break;
        default: return fail(c, ST_E_UNSUPPORTED, "this operand has a derivative in a pair only");
    }
    LineArgsT<T> a = make_args<T>(c, dir);
    set_d1(c, a, 0, asym, iadd, cadd);
    a.k0 = F.k0; a.k1 = F.k1; a.k2 = F.k2;
    // the derivative of a*b with half the factor, plus that of c
    if (F.op == PR_MULPLUS) { a.op[1] = a.op[0]; a.op[1].fac1 = 0.5 * a.op[0].fac1; }
    const T *in[4] = {F.a, F.b, F.c, F.d};
    for (int k = 0; k < nin; k++) ST_TRY(aligned(c, in[k]));
    ST_TRY(aligned(c, dF));
    return launch(c, id, a, in, &dF);
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
// two launches.  A pair of other operands that have one of their own runs as
// two launches.
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

}  // namespace st
