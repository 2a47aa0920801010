// Entry points nk_unary (the 23 activations + AssignLeft's copy) and nk_scalar_binary (tensor op scalar).
// Compiled with -fmad=false (see nk_scalarfun.cuh).

#include "nk_ew_kernels.cuh"

using namespace nkew;

namespace {

#define NK_UNARY_CASE(FUN, DER) \
    case (FUN * 2 + (DER ? 1 : 0)): return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, UnaryFix<T, FUN, DER>{});

// the common activations get compile-time functors (forward; tanh / sig / relu also their derivative)
template <class T>
int launch_unary(nk_ctx* ctx, int fun, bool derive, T* out, const T* in, const EwPlan& p) {
    switch (fun * 2 + (derive ? 1 : 0)) {
        NK_UNARY_CASE(NK_FUN_IDY, false) NK_UNARY_CASE(NK_FUN_RELU, false) NK_UNARY_CASE(NK_FUN_TANH, false) NK_UNARY_CASE(NK_FUN_SIG, false)
        NK_UNARY_CASE(NK_FUN_ABS, false) NK_UNARY_CASE(NK_FUN_QUAD, false) NK_UNARY_CASE(NK_FUN_EXP, false) NK_UNARY_CASE(NK_FUN_GELU, false)
        NK_UNARY_CASE(NK_FUN_SILU, false) NK_UNARY_CASE(NK_FUN_SOFTPLUS, false)
        NK_UNARY_CASE(NK_FUN_TANH, true) NK_UNARY_CASE(NK_FUN_SIG, true) NK_UNARY_CASE(NK_FUN_RELU, true)
        default: break;
    }
    return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, UnaryF<T>{fun, derive});
}

template <class T>
int launch_scalar(nk_ctx* ctx, int op, int d, T value, T* out, const T* in, const EwPlan& p) {
    if (d < 0) {
        switch (op) {
            case NK_OP_ADD: return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, ScalarFix<T, NK_OP_ADD>{value});
            case NK_OP_SUB: return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, ScalarFix<T, NK_OP_SUB>{value});
            case NK_OP_MUL: return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, ScalarFix<T, NK_OP_MUL>{value});
            case NK_OP_DIV: return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, ScalarFix<T, NK_OP_DIV>{value});
            default: break;
        }
    }
    return launch_ew<T, 1>(ctx, out, in, (const T*)nullptr, p, ScalarF<T>{op, d, value});
}

// f and f' of a contiguous tensor in one pass. The eager derivative of a function is taken where its value is, and costs another
// read of the input and, for the exponential ones, the whole exponential again; here the compiler shares it between the two. The
// next vector is requested before this one's arithmetic, as in nk_ew_linear_kernel. tanh over 2^26 F32: its F64 arithmetic (about
// 135 us) and 12 bytes per element (121 us) bound the pass, which takes 170; the two separate ones took 136 + 150.
template <class T, class F0, class F1>
__global__ void __launch_bounds__(256) nk_ew_both_kernel(T* out, T* der, const T* a, int64_t n, F0 f0, F1 f1) {   // (either drain may be the source)
    using V = typename Vec4<T>::type;
    constexpr int N = Vec4<T>::N;
    const int64_t nvec = n / N, stride = int64_t(gridDim.x) * blockDim.x, tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    V cur, nxt;
    if (tid < nvec) cur = __ldcs(reinterpret_cast<const V*>(a) + tid);
    for (int64_t i = tid; i < nvec; i += stride) {
        if (i + stride < nvec) nxt = __ldcs(reinterpret_cast<const V*>(a) + i + stride);
        T ov[N], dv[N];
        apply_vec<T, N, 1>(f0, reinterpret_cast<const T*>(&cur), static_cast<const T*>(nullptr), ov);
        apply_vec<T, N, 1>(f1, reinterpret_cast<const T*>(&cur), static_cast<const T*>(nullptr), dv);
        __stcs(reinterpret_cast<V*>(out) + i, *reinterpret_cast<V*>(ov));
        __stcs(reinterpret_cast<V*>(der) + i, *reinterpret_cast<V*>(dv));
        cur = nxt;
    }
    for (int64_t i = nvec * N + tid; i < n; i += stride) {
        const T x = a[i];
        out[i] = f0(x, T(0));
        der[i] = f1(x, T(0));
    }
}
template <class T, class F0, class F1>
int launch_both(nk_ctx* ctx, T* out, T* der, const T* a, int64_t n, F0 f0, F1 f1) {
    const int grid = nk_grid_for(ctx, (n + Vec4<T>::N - 1) / Vec4<T>::N, 256, 8);
    nk_ew_both_kernel<T, F0, F1><<<grid, 256, 0, ctx->stream>>>(out, der, a, n, f0, f1);
    return nk_after_launch(ctx, "nk_ew_both_kernel");
}
template <class T>
int unary_both(nk_ctx* ctx, int fun, T* out, T* der, const T* in, const EwPlan& p, const EwPlan& pd) {
    // one pass where all three run along one dense dim with 16-byte accesses, otherwise two launches
    const bool dense = p.row_major && pd.row_major && p.nd == 1 && pd.nd == 1 && p.s0[0] == 1 && p.s1[0] == 1 && pd.s0[0] == 1 &&
                       aligned16(out + p.b0) && aligned16(in + p.b1) && aligned16(der + pd.b0);
    if (!dense) {
        // the drain that is the source itself is written last
        const bool derivative_last = der + pd.b0 == in + pd.b1;
        if (derivative_last) {
            const int st = launch_unary<T>(ctx, fun, false, out, in, p);
            return st ? st : launch_unary<T>(ctx, fun, true, der, in, pd);
        }
        const int st = launch_unary<T>(ctx, fun, true, der, in, pd);
        return st ? st : launch_unary<T>(ctx, fun, false, out, in, p);
    }
    out += p.b0; der += pd.b0; in += p.b1;
#define NK_BOTH_CASE(FUN) case FUN: return launch_both<T>(ctx, out, der, in, p.total, UnaryFix<T, FUN, false>{}, UnaryFix<T, FUN, true>{});
    switch (fun) {
        NK_BOTH_CASE(NK_FUN_TANH) NK_BOTH_CASE(NK_FUN_SIG) NK_BOTH_CASE(NK_FUN_SILU) NK_BOTH_CASE(NK_FUN_GELU) NK_BOTH_CASE(NK_FUN_RELU)
        NK_BOTH_CASE(NK_FUN_SOFTPLUS)
        default: break;
    }
#undef NK_BOTH_CASE
    return launch_both<T>(ctx, out, der, in, p.total, UnaryF<T>{fun, false}, UnaryF<T>{fun, true});
}

}  // namespace

extern "C" int nk_unary_both(nk_ctx* ctx, int32_t fun, int32_t dtype, int32_t rank, nk_buf* drn, const int32_t* cfg0, nk_buf* ddrn, const int32_t* cfgd,
                             nk_buf* src, const int32_t* cfg1) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_unary_both: dtype %d not supported (F32/F64 only)", dtype);
    if (fun < 0 || fun >= NK_FUN_COUNT) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_unary_both: unknown function id %d", fun);
    NkView v0, vd, v1;
    int st;
    if ((st = nk_view_parse(ctx, "nk_unary_both(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    if ((st = nk_view_parse(ctx, "nk_unary_both(derivative drain)", ddrn, cfgd, rank, dtype, &vd))) return st;
    if ((st = nk_view_parse(ctx, "nk_unary_both(src)", src, cfg1, rank, dtype, &v1))) return st;
    for (int k = 0; k < rank; k++)
        if (v0.shape[k] != v1.shape[k] || vd.shape[k] != v1.shape[k])
            return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_unary_both: shapes differ at dim %d (%lld, %lld vs %lld)", k, (long long)v0.shape[k],
                           (long long)vd.shape[k], (long long)v1.shape[k]);
    EwPlan p, pd;
    make_plan(v0, &v1, nullptr, nullptr, nullptr, &p);
    make_plan(vd, &v1, nullptr, nullptr, nullptr, &pd);
    if (dtype == NK_F32) return unary_both<float>(ctx, fun, data_of<float>(drn), data_of<float>(ddrn), data_of<float>(src), p, pd);
    return unary_both<double>(ctx, fun, data_of<double>(drn), data_of<double>(ddrn), data_of<double>(src), p, pd);
}

extern "C" int nk_unary(nk_ctx* ctx, int32_t fun, int32_t dtype, int32_t rank,
                        nk_buf* drn, const int32_t* cfg0, nk_buf* src, const int32_t* cfg1, int32_t d) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_unary: dtype %d not supported (F32/F64 only)", dtype);
    if (fun < 0 || fun >= NK_FUN_COUNT) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_unary: unknown function id %d", fun);
    NkView v0, v1;
    int st;
    if ((st = nk_view_parse(ctx, "nk_unary(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    if ((st = nk_view_parse(ctx, "nk_unary(src)", src, cfg1, rank, dtype, &v1))) return st;
    for (int k = 0; k < rank; k++)
        if (v0.shape[k] != v1.shape[k])
            return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_unary: shapes differ at dim %d (%lld vs %lld)", k, (long long)v0.shape[k], (long long)v1.shape[k]);
    EwPlan p;
    make_plan(v0, &v1, nullptr, nullptr, nullptr, &p);
    if (dtype == NK_F32) return launch_unary<float>(ctx, fun, d >= 0, data_of<float>(drn), data_of<float>(src), p);
    return launch_unary<double>(ctx, fun, d >= 0, data_of<double>(drn), data_of<double>(src), p);
}

extern "C" int nk_scalar_binary(nk_ctx* ctx, int32_t op, int32_t dtype, int32_t rank,
                                nk_buf* drn, const int32_t* cfg0, nk_buf* src, const int32_t* cfg1, double value, int32_t d) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_scalar_binary: dtype %d not supported (F32/F64 only)", dtype);
    if (!known_op(op, true, false)) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_scalar_binary: unknown op %d", op);
    NkView v0, v1;
    int st;
    if ((st = nk_view_parse(ctx, "nk_scalar_binary(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    if ((st = nk_view_parse(ctx, "nk_scalar_binary(src)", src, cfg1, rank, dtype, &v1))) return st;
    for (int k = 0; k < rank; k++)
        if (v0.shape[k] != v1.shape[k])
            return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_scalar_binary: shapes differ at dim %d (%lld vs %lld)", k, (long long)v0.shape[k], (long long)v1.shape[k]);
    EwPlan p;
    make_plan(v0, &v1, nullptr, nullptr, nullptr, &p);
    int dd = d < 0 ? -1 : d;
    if (dtype == NK_F32) return launch_scalar<float>(ctx, op, dd, float(value), data_of<float>(drn), data_of<float>(src), p);
    return launch_scalar<double>(ctx, op, dd, value, data_of<double>(drn), data_of<double>(src), p);
}

