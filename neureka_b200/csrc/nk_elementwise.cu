// Entry points nk_broadcast, nk_binary, nk_fill_fun, nk_sum and the backward-broadcast reduction kernel.
// (nk_unary and nk_scalar_binary live in nk_ew_unary.cu; the forward kernels in nk_ew_kernels.cuh.)
//
// Compiled with -fmad=false (see nk_scalarfun.cuh).

#include "nk_ew_kernels.cuh"
#include "nk_launch_rules.h"
#include "nk_ptx.cuh"

using namespace nkew;

namespace {

// forward + - * / with compile-time functors, everything else through the run-time functor
template <class T, int FAMILY>
int launch_binary(nk_ctx* ctx, int op, int d, T* out, const T* a, const T* b, const EwPlan& p) {
    if (d < 0) {
        switch (op) {
            case NK_OP_ADD: return launch_ew<T, 2>(ctx, out, a, b, p, BinFix<T, NK_OP_ADD>{});
            case NK_OP_SUB: return launch_ew<T, 2>(ctx, out, a, b, p, BinFix<T, NK_OP_SUB>{});
            case NK_OP_MUL: return launch_ew<T, 2>(ctx, out, a, b, p, BinFix<T, NK_OP_MUL>{});
            case NK_OP_DIV: return launch_ew<T, 2>(ctx, out, a, b, p, BinFix<T, NK_OP_DIV>{});
            default: break;
        }
    }
    return launch_ew<T, 2>(ctx, out, a, b, p, BinF<T, FAMILY>{op, d});
}

// One term of the backward-broadcast sum, added to 0 like a sum of one element (the sign of a zero differs from the bare term).
template <class T, int OP, int D> struct TermFix {
    __device__ __forceinline__ T operator()(T a, T b) const { return T(0) + nkf::bin<0>(OP, D, a, b); }
};
template <class T> struct TermF {
    int op, d;
    __device__ __forceinline__ T operator()(T a, T b) const { return T(0) + nkf::bin<0>(op, d, a, b); }
};
template <class T>
int launch_term(nk_ctx* ctx, int op, int d, T* out, const T* a, const T* b, const EwPlan& p) {
    if (op == NK_OP_ADD) return launch_ew<T, 2>(ctx, out, a, b, p, TermFix<T, NK_OP_ADD, 0>{});
    if (op == NK_OP_MUL_BOTH) return launch_ew<T, 2>(ctx, out, a, b, p, TermFix<T, NK_OP_MUL_BOTH, 0>{});
    return launch_ew<T, 2>(ctx, out, a, b, p, TermF<T>{op, d});
}

// ---- broadcast backward: reduction over the dims where the origin is smaller -------------------------
struct RedPlan {
    int rank;
    int64_t total;                  // origin elements
    int64_t odiv[NK_MAX_RANK];      // decode of the origin's flat index
    int64_t s0[NK_MAX_RANK];        // origin strides
    int64_t p1[NK_MAX_RANK], p2[NK_MAX_RANK];  // handle/drain stride applied to the origin index
    int nred;
    int64_t rext[NK_MAX_RANK], r1[NK_MAX_RANK], r2[NK_MAX_RANK];  // reduced dims: extent, handle stride, drain stride
    int64_t b0, b1, b2;
};

// One thread per origin element; the reduction runs with the lowest reduced dim fastest, the order of
// the state machine in CPUBroadcast.java:118-150, so F32 results match the CPU bit for bit.
template <class T>
__global__ void __launch_bounds__(256) nk_broadcast_reduce_kernel(T* __restrict__ t0, const T* __restrict__ t1, const T* __restrict__ t2,
                                                                  RedPlan p, int op, int d) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < p.total; i += stride) {
        int64_t rem = i, o0 = p.b0, o1 = p.b1, o2 = p.b2;
        for (int k = 0; k < p.rank; k++) {
            int64_t idx = rem / p.odiv[k];
            rem -= idx * p.odiv[k];
            o0 += idx * p.s0[k]; o1 += idx * p.p1[k]; o2 += idx * p.p2[k];
        }
        T value = 0;
        if (p.nred == 1) {   // (at least one dim is reduced: nothing reduced is an elementwise call)
            for (int64_t r = 0; r < p.rext[0]; r++) value += nkf::bin<0>(op, d, t1[o1 + r * p.r1[0]], t2[o2 + r * p.r2[0]]);
        } else {
            int64_t q[NK_MAX_RANK];
            for (int k = 0; k < p.nred; k++) q[k] = 0;
            int64_t c1 = o1, c2 = o2;
            while (true) {
                value += nkf::bin<0>(op, d, t1[c1], t2[c2]);
                int k = 0;
                for (; k < p.nred; k++) {
                    q[k]++; c1 += p.r1[k]; c2 += p.r2[k];
                    if (q[k] < p.rext[k]) break;
                    c1 -= q[k] * p.r1[k]; c2 -= q[k] * p.r2[k]; q[k] = 0;
                }
                if (k == p.nred) break;
            }
        }
        t0[o0] = value;
    }
}

// Vectorised variant: the innermost dim is not reduced and the drain and the origin are unit-stride along it, so a thread owns
// W neighbouring origin elements (a 128-bit vector, or one element where extents or alignments are odd: lanes still run
// along contiguous memory) and every step of its reduction loop is one load per operand. What bounds it is the latency of
// those loads -- the origin is small, so there are few threads -- hence STEPS steps are requested ahead of the (ordered)
// additions. The summation order per element is unchanged (lowest reduced dim fastest), hence still bit-identical to the
// CPU for + - *. OP/D are compile-time for the common operators. HMODE: the handle is one value per step (0), runs along with
// the origin (1), or does not move along the lowest reduced dim at all and is read once per outer step (2: one value, the
// zero handle of a sum's or difference's backward pass).
template <class T, int W> struct VecOf { using type = T; };
template <> struct VecOf<float, 4> { using type = float4; };
template <> struct VecOf<double, 2> { using type = double2; };
template <class T, int W, int OP, int D, int HMODE>
__global__ void __launch_bounds__(128) nk_broadcast_reduce_vec_kernel(T* __restrict__ t0, const T* __restrict__ t1, const T* __restrict__ t2,
                                                                      RedPlan p, int64_t total_vec) {
    using V = typename VecOf<T, W>::type;
    constexpr int STEPS = 8;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t v = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < total_vec; v += stride) {
        int64_t rem = v * W, o0 = p.b0, o1 = p.b1, o2 = p.b2;
        for (int k = 0; k < p.rank; k++) {
            int64_t idx = rem / p.odiv[k];
            rem -= idx * p.odiv[k];
            o0 += idx * p.s0[k]; o1 += idx * p.p1[k]; o2 += idx * p.p2[k];
        }
        T acc[W];
#pragma unroll
        for (int k = 0; k < W; k++) acc[k] = T(0);
        int64_t q[NK_MAX_RANK];
        for (int k = 0; k < p.nred; k++) q[k] = 0;
        const int64_t n0 = p.nred > 0 ? p.rext[0] : 1, a0 = p.nred > 0 ? p.r1[0] : 0, b0 = p.nred > 0 ? p.r2[0] : 0;
        int64_t c1 = o1, c2 = o2;
        while (true) {
            const T h_fixed = HMODE == 2 ? t1[c1] : T(0);
            const T *h_ptr = t1 + c1, *d_ptr = t2 + c2;
            int64_t r = 0;
            for (; r + STEPS <= n0; r += STEPS) {
                T hv[STEPS][W], dv[STEPS][W];
#pragma unroll
                for (int u = 0; u < STEPS; u++) {
                    *reinterpret_cast<V*>(dv[u]) = __ldcs(reinterpret_cast<const V*>(d_ptr));
                    if (HMODE == 1) *reinterpret_cast<V*>(hv[u]) = __ldg(reinterpret_cast<const V*>(h_ptr));
                    else if (HMODE == 0) hv[u][0] = __ldg(h_ptr);
                    d_ptr += b0;
                    h_ptr += a0;
                }
#pragma unroll
                for (int u = 0; u < STEPS; u++)
#pragma unroll
                    for (int k = 0; k < W; k++)
                        acc[k] += nkf::bin<0>(OP, D, HMODE == 1 ? hv[u][k] : HMODE == 0 ? hv[u][0] : h_fixed, dv[u][k]);
            }
            for (; r < n0; r++) {
                T hv[W], dv[W];
                *reinterpret_cast<V*>(dv) = __ldcs(reinterpret_cast<const V*>(d_ptr));
                if (HMODE == 1) *reinterpret_cast<V*>(hv) = __ldg(reinterpret_cast<const V*>(h_ptr));
                else hv[0] = HMODE == 0 ? __ldg(h_ptr) : h_fixed;
                d_ptr += b0;
                h_ptr += a0;
#pragma unroll
                for (int k = 0; k < W; k++) acc[k] += nkf::bin<0>(OP, D, HMODE == 1 ? hv[k] : hv[0], dv[k]);
            }
            int k = 1;
            for (; k < p.nred; k++) {
                q[k]++; c1 += p.r1[k]; c2 += p.r2[k];
                if (q[k] < p.rext[k]) break;
                c1 -= q[k] * p.r1[k]; c2 -= q[k] * p.r2[k]; q[k] = 0;
            }
            if (k >= p.nred) break;
        }
        *reinterpret_cast<V*>(t0 + o0) = *reinterpret_cast<V*>(acc);
    }
}

template <class T, int W, int HMODE>
bool launch_reduce_vec(nk_ctx* ctx, T* t0, const T* t1, const T* t2, const RedPlan& p, int op, int d, int* status) {
    const int64_t total_vec = p.total / W;
    const int block = 128, grid = nk_grid_for(ctx, total_vec, block, 16);
#define NK_RED(OPC, DC) nk_broadcast_reduce_vec_kernel<T, W, OPC, DC, HMODE><<<grid, block, 0, ctx->stream>>>(t0, t1, t2, p, total_vec)
    if (op == NK_OP_MUL_BOTH) NK_RED(NK_OP_MUL_BOTH, 0);
    else if (op == NK_OP_ADD) NK_RED(NK_OP_ADD, 0);
    else if (op == NK_OP_SUB && d == 0) NK_RED(NK_OP_SUB, 0);
    else if (op == NK_OP_SUB && d == 1) NK_RED(NK_OP_SUB, 1);
    else if (op == NK_OP_MUL && d == 0) NK_RED(NK_OP_MUL, 0);
    else if (op == NK_OP_MUL && d == 1) NK_RED(NK_OP_MUL, 1);
    else return false;
#undef NK_RED
    *status = nk_after_launch(ctx, "nk_broadcast_reduce_vec_kernel");
    return true;
}

template <class T>
bool try_reduce_vec(nk_ctx* ctx, T* t0, const T* t1, const T* t2, const RedPlan& p, int op, int d, const NkView& v0, int* status) {
    constexpr int N = Vec4<T>::N;
    const int last = p.rank - 1;
    if (p.nred < 1 || !v0.imap_row_major) return false;
    // innermost dim: kept (not reduced), unit stride in origin and drain, unit or zero stride in the handle
    if (p.s0[last] != 1 || p.p2[last] != 1 || (p.p1[last] != 1 && p.p1[last] != 0)) return false;
    const bool along = p.p1[last] == 1, fixed = !along && p.r1[0] == 0;
    // whole 128-bit vectors: extents, strides and addresses allow them for every access (the handle's only if it runs along)
    auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    bool vec = v0.shape[last] % N == 0 && al(t0 + p.b0) && al(t2 + p.b2) && (!along || al(t1 + p.b1));
    for (int k = 0; k < last; k++)
        if (p.s0[k] % N || p.p2[k] % N || (along && p.p1[k] % N)) vec = false;
    for (int k = 0; k < p.nred; k++)
        if (p.r2[k] % N || (along && p.r1[k] % N)) vec = false;
    if (vec) {
        if (along) return launch_reduce_vec<T, N, 1>(ctx, t0, t1, t2, p, op, d, status);
        if (fixed) return launch_reduce_vec<T, N, 2>(ctx, t0, t1, t2, p, op, d, status);
        return launch_reduce_vec<T, N, 0>(ctx, t0, t1, t2, p, op, d, status);
    }
    if (v0.shape[last] < 32) return false;   // single elements per lane: worth it where a warp runs along the innermost dim
    if (along) return launch_reduce_vec<T, 1, 1>(ctx, t0, t1, t2, p, op, d, status);
    if (fixed) return launch_reduce_vec<T, 1, 2>(ctx, t0, t1, t2, p, op, d, status);
    return launch_reduce_vec<T, 1, 0>(ctx, t0, t1, t2, p, op, d, status);
}

// ---- fill with fun(value) ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(256) nk_fill_fun_kernel(T* __restrict__ out, EwPlan p, int fun, bool derive, T value) {
    const T v = nkf::fun(fun, derive, value);
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < p.total; i += stride) {
        int64_t rem = i, o0 = p.b0;
        for (int k = 0; k < p.nd; k++) {
            int64_t idx = rem / p.div[k];
            rem -= idx * p.div[k];
            o0 += idx * p.s0[k];
        }
        out[o0] = v;
    }
}

// ---- sum: 128-wide tiles, recursively, in CPUSum's order ----------------------------------------------
// The 128 elements of a tile are added in index order by one lane, so the work is turned through shared memory:
//   * nk_sum_rows_kernel (contiguous, 16-byte aligned): a warp requests 32 whole tiles with 16-byte asynchronous copies, into rows
//     padded by 16 bytes, and lane t then adds row t. The copies need no registers: twelve warps' 16 KB each are in flight per
//     SM. 2^26 F32 elements: 46 us (40 is the floor); one tile per warp, one lane adding: 487.
//   * nk_sum_tiles_kernel (any view, many tiles): the same through registers, 16 elements of every tile at a time.
//   * nk_sum_warp_kernel (any view): a tile per warp, staged by all lanes and added by one -- a thirty-second of the adders, but 32 times
//     the warps, which is what fewer tiles than the chip has lanes need (1000 x 1000 F32, a slice: 20 us, in groups of 32 tiles 83).
//   * nk_sum_last_kernel: at most 32 tiles, i.e. the last two levels of any sum (or all of a sum of up to 2^12 elements) in
//     one CTA: a warp stages a tile, one lane adds it; one lane then adds the tile sums.
struct SumView {
    int nd;                       // merged dims (0: contiguous, from the pointer on; not for nk_sum_tiles_kernel)
    int64_t div[NK_MAX_RANK], s[NK_MAX_RANK];
    int64_t base;
};
__device__ __forceinline__ int64_t sum_offset(const SumView& v, int64_t i) {
    int64_t src = v.base;
    for (int j = 0; j < v.nd; j++) { const int64_t idx = i / v.div[j]; i -= idx * v.div[j]; src += idx * v.s[j]; }
    return src;
}
__device__ __forceinline__ int64_t sum_place(const SumView& v, int64_t i) { return v.nd == 0 ? i : sum_offset(v, i); }
template <class T> struct SumRows {
    static constexpr int VPT = 128 * int(sizeof(T)) / 16;        // 16-byte vectors per tile
    static constexpr int PITCH = 128 + 16 / int(sizeof(T));      // elements per padded row
    static constexpr int WARPS = sizeof(T) == 4 ? 4 : 2;
    static constexpr int SMEM = WARPS * 32 * PITCH * int(sizeof(T));
};
template <class T>
__global__ void __launch_bounds__(SumRows<T>::WARPS * 32) nk_sum_rows_kernel(const T* __restrict__ in, int64_t n, T* __restrict__ out, int64_t n_tiles) {
    using C = SumRows<T>;
    using V = typename Vec4<T>::type;
    constexpr int N = Vec4<T>::N;
    extern __shared__ __align__(16) unsigned char sum_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* rows = reinterpret_cast<T*>(sum_smem) + warp * 32 * C::PITCH;
    const int64_t groups = (n_tiles + 31) / 32;
    for (int64_t g = int64_t(blockIdx.x) * C::WARPS + warp; g < groups; g += int64_t(gridDim.x) * C::WARPS) {
        const int64_t first = g * 4096;
        const int64_t left = n - first;
        const int count = left < 4096 ? int(left) : 4096;        // elements of this group
        const int whole = count / N;                             // whole vectors of it; the rest one by one
        for (int v = lane; v < 32 * C::VPT; v += 32) {
            T* dst = rows + (v / C::VPT) * C::PITCH + (v % C::VPT) * N;
            if (v < whole) nk_cp_async_16(dst, in + first + v * N, 16);
            else
                for (int e = 0; e < N; e++)
                    if (v * N + e < count) dst[e] = in[first + v * N + e];
        }
        nk_cp_async_commit();
        nk_cp_async_wait<0>();
        __syncwarp();
        const int len = count - lane * 128 < 128 ? count - lane * 128 : 128;
        if (len > 0) {
            const T* row = rows + lane * C::PITCH;
            T value = 0;
            if (len == 128) {
#pragma unroll 8
                for (int c = 0; c < 128; c += N) {
                    T e[N];
                    *reinterpret_cast<V*>(e) = *reinterpret_cast<const V*>(row + c);
#pragma unroll
                    for (int k = 0; k < N; k++) value += e[k];
                }
            } else {
                for (int c = 0; c < len; c++) value += row[c];
            }
            out[g * 32 + lane] = value;
        }
        __syncwarp();
    }
}
template <class T>
__global__ void __launch_bounds__(128) nk_sum_tiles_kernel(const T* __restrict__ in, const SumView v, int64_t n, T* __restrict__ out, int64_t n_tiles) {
    constexpr int C = 16, STEPS = 128 / C, PER = 32 / C;   // elements of a tile per step; lanes 0..C-1 load one tile, C..2C-1 the next
    __shared__ T stage[4][32][C + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sub = lane / C, col = lane % C;
    const int64_t groups = (n_tiles + 31) / 32;
    for (int64_t g = int64_t(blockIdx.x) * 4 + warp; g < groups; g += int64_t(gridDim.x) * 4) {
        const int64_t first = g * 4096;
        T val[32 / PER];
        auto load = [&](int step) {
#pragma unroll
            for (int k = 0; k < 32 / PER; k++) {
                const int64_t i = first + (k * PER + sub) * 128 + step * C + col;
                val[k] = in[sum_offset(v, i < n ? i : n - 1)];   // past the end: never added
            }
        };
        load(0);
        const int64_t mine = first + lane * 128;      // this lane's tile
        const int len = mine >= n ? 0 : (n - mine < 128 ? int(n - mine) : 128);
        T value = 0;
        for (int step = 0; step < STEPS; step++) {
#pragma unroll
            for (int k = 0; k < 32 / PER; k++) stage[warp][k * PER + sub][col] = val[k];
            __syncwarp();
            if (step + 1 < STEPS) load(step + 1);
            if (len == 128) {
#pragma unroll
                for (int c = 0; c < C; c++) value += stage[warp][lane][c];
            } else {
                for (int c = 0; c < C; c++)
                    if (step * C + c < len) value += stage[warp][lane][c];
            }
            __syncwarp();
        }
        if (len > 0) out[g * 32 + lane] = value;
    }
}
template <class T>
__global__ void __launch_bounds__(128) nk_sum_warp_kernel(const T* __restrict__ in, const SumView v, int64_t n, T* __restrict__ out, int64_t n_tiles) {
    __shared__ T tile[4][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int64_t t = int64_t(blockIdx.x) * 4 + warp; t < n_tiles; t += int64_t(gridDim.x) * 4) {
        const int64_t off = t * 128;
        const int lim = off + 128 < n ? 128 : int(n - off);
        for (int k = lane; k < lim; k += 32) tile[warp][k] = in[sum_place(v, off + k)];
        __syncwarp();
        if (lane == 0) {
            T value = 0;
            for (int k = 0; k < lim; k++) value += tile[warp][k];
            out[t] = value;
        }
        __syncwarp();
    }
}
template <class T>
__global__ void __launch_bounds__(1024) nk_sum_last_kernel(const T* __restrict__ in, const SumView v, int n, T* __restrict__ out) {
    __shared__ T tile[NK_SUM_LAST / 128][128];
    __shared__ T part[NK_SUM_LAST / 128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, off = warp * 128;   // a warp per tile
    const int lim = off + 128 < n ? 128 : n - off;
    for (int k = lane; k < lim; k += 32) tile[warp][k] = in[sum_place(v, off + k)];
    __syncwarp();
    if (lane == 0) {
        T value = 0;
        for (int k = 0; k < lim; k++) value += tile[warp][k];
        part[warp] = value;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // a single tile is the result; several are one more tile, added in order from 0
        const int n_tiles = int(blockDim.x >> 5);
        T value = 0;
        if (n_tiles == 1) value = part[0];
        else for (int k = 0; k < n_tiles; k++) value += part[k];
        *out = value;
    }
}

}  // namespace

// ------------------------------------------------------------------------------------------------
// entry points
// ------------------------------------------------------------------------------------------------
extern "C" int nk_broadcast(nk_ctx* ctx, int32_t op, int32_t dtype, int32_t rank,
                            nk_buf* drn, const int32_t* cfg0, nk_buf* a, const int32_t* cfg1, nk_buf* b, const int32_t* cfg2,
                            int32_t d) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64)  // CPUBroadcast.java:46-56 supports exactly these two
        return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_broadcast: dtype %d not supported (F32/F64 only)", dtype);
    if (!known_op(op, false, true)) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast: unknown op %d", op);
    NkView v0, v1, v2;
    int st;
    if ((st = nk_view_parse(ctx, "nk_broadcast(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    if ((st = nk_view_parse(ctx, "nk_broadcast(src1)", a, cfg1, rank, dtype, &v1))) return st;
    if ((st = nk_view_parse(ctx, "nk_broadcast(src2)", b, cfg2, rank, dtype, &v2))) return st;
    if (d < 0) {
        bool f1[NK_MAX_RANK], f2[NK_MAX_RANK];
        for (int k = 0; k < rank; k++) {
            // CPUBroadcast.java:82-93: equal shapes -> both follow; otherwise the larger follows, the smaller stays at 0
            f1[k] = v1.shape[k] >= v2.shape[k];
            f2[k] = v2.shape[k] >= v1.shape[k];
            int64_t big = v1.shape[k] > v2.shape[k] ? v1.shape[k] : v2.shape[k];
            if (v0.shape[k] > big)
                return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast: drain dim %d = %lld exceeds both sources (%lld, %lld)", k,
                               (long long)v0.shape[k], (long long)v1.shape[k], (long long)v2.shape[k]);
        }
        EwPlan p;
        make_plan(v0, &v1, f1, &v2, f2, &p);
        if (dtype == NK_F32) return launch_binary<float, 0>(ctx, op, -1, data_of<float>(drn), data_of<float>(a), data_of<float>(b), p);
        return launch_binary<double, 0>(ctx, op, -1, data_of<double>(drn), data_of<double>(a), data_of<double>(b), p);
    }
    // d >= 0: (origin t0, handle t1, drain t2), CPUBroadcast.java:99-158
    if (d > 1) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast: derivative index %d, expected 0 or 1", d);
    RedPlan p;
    p.rank = rank;
    p.total = v0.size;
    p.nred = 0;
    p.b0 = v0.base; p.b1 = v1.base; p.b2 = v2.base;
    for (int k = 0; k < rank; k++) {
        p.odiv[k] = v0.imap[k];
        p.s0[k] = v0.estride[k];
        int64_t s0 = v0.shape[k], s1 = v1.shape[k], s2 = v2.shape[k];
        if (s0 == s1) {
            if (s2 != 1 && s2 < s0)
                return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast(d>=0): dim %d: drain extent %lld smaller than origin %lld", k, (long long)s2, (long long)s0);
            p.p1[k] = v1.estride[k];
            p.p2[k] = (s2 == 1) ? 0 : v2.estride[k];
        } else if (s0 > s1) {
            if (s2 < s0) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast(d>=0): dim %d: drain extent %lld smaller than origin %lld", k, (long long)s2, (long long)s0);
            p.p1[k] = 0;
            p.p2[k] = v2.estride[k];
        } else {  // s0 < s1: summed over the handle's extent, handle and drain advance together
            if (s0 != 1) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_broadcast(d>=0): dim %d: origin extent %lld must be 1 where the handle (%lld) is larger", k, (long long)s0, (long long)s1);
            if (s2 < s1) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_broadcast(d>=0): dim %d: drain extent %lld smaller than handle %lld", k, (long long)s2, (long long)s1);
            p.p1[k] = 0; p.p2[k] = 0;
            p.rext[p.nred] = s1; p.r1[p.nred] = v1.estride[k]; p.r2[p.nred] = v2.estride[k];
            p.nred++;
        }
    }
    if (p.nred == 0) {
        // nothing is summed (the origin has the error's shape): an elementwise pass, with the reduction's 0 + term
        bool f1[NK_MAX_RANK], f2[NK_MAX_RANK];
        for (int k = 0; k < rank; k++) {
            f1[k] = v0.shape[k] == v1.shape[k];
            f2[k] = !f1[k] || v2.shape[k] != 1;
        }
        EwPlan e;
        make_plan(v0, &v1, f1, &v2, f2, &e);
        if (dtype == NK_F32) return launch_term<float>(ctx, op, d, data_of<float>(drn), data_of<float>(a), data_of<float>(b), e);
        return launch_term<double>(ctx, op, d, data_of<double>(drn), data_of<double>(a), data_of<double>(b), e);
    }
    {
        int vst = NK_OK;
        bool done = (dtype == NK_F32) ? try_reduce_vec<float>(ctx, data_of<float>(drn), data_of<float>(a), data_of<float>(b), p, op, d, v0, &vst)
                                      : try_reduce_vec<double>(ctx, data_of<double>(drn), data_of<double>(a), data_of<double>(b), p, op, d, v0, &vst);
        if (done) return vst;
    }
    int block = 256, grid = nk_grid_for(ctx, p.total, block, 8);
    if (dtype == NK_F32) nk_broadcast_reduce_kernel<float><<<grid, block, 0, ctx->stream>>>(data_of<float>(drn), data_of<float>(a), data_of<float>(b), p, op, d);
    else nk_broadcast_reduce_kernel<double><<<grid, block, 0, ctx->stream>>>(data_of<double>(drn), data_of<double>(a), data_of<double>(b), p, op, d);
    return nk_after_launch(ctx, "nk_broadcast_reduce_kernel");
}

extern "C" int nk_binary(nk_ctx* ctx, int32_t op, int32_t dtype, int32_t rank,
                         nk_buf* drn, const int32_t* cfg0, nk_buf* a, const int32_t* cfg1, nk_buf* b, const int32_t* cfg2,
                         int32_t d) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_binary: dtype %d not supported (F32/F64 only)", dtype);
    if (!known_op(op, false, false)) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_binary: unknown op %d", op);
    NkView v0, v1, v2;
    int st;
    if ((st = nk_view_parse(ctx, "nk_binary(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    if ((st = nk_view_parse(ctx, "nk_binary(src1)", a, cfg1, rank, dtype, &v1))) return st;
    if ((st = nk_view_parse(ctx, "nk_binary(src2)", b, cfg2, rank, dtype, &v2))) return st;
    for (int k = 0; k < rank; k++)
        if (v0.shape[k] != v1.shape[k] || v0.shape[k] != v2.shape[k])
            return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_binary: shapes differ at dim %d (%lld, %lld, %lld)", k,
                           (long long)v0.shape[k], (long long)v1.shape[k], (long long)v2.shape[k]);
    EwPlan p;
    make_plan(v0, &v1, nullptr, &v2, nullptr, &p);
    int dd = d < 0 ? -1 : d;
    if (dtype == NK_F32) return launch_binary<float, 1>(ctx, op, dd, data_of<float>(drn), data_of<float>(a), data_of<float>(b), p);
    return launch_binary<double, 1>(ctx, op, dd, data_of<double>(drn), data_of<double>(a), data_of<double>(b), p);
}

extern "C" int nk_fill_fun(nk_ctx* ctx, int32_t fun, int32_t dtype, int32_t rank, nk_buf* drn, const int32_t* cfg0,
                           double value, int32_t d) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_fill_fun: dtype %d not supported (F32/F64 only)", dtype);
    if (fun < 0 || fun >= NK_FUN_COUNT) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_fill_fun: unknown function id %d", fun);
    NkView v0;
    int st;
    if ((st = nk_view_parse(ctx, "nk_fill_fun(drain)", drn, cfg0, rank, dtype, &v0))) return st;
    EwPlan p;
    make_plan(v0, nullptr, nullptr, nullptr, nullptr, &p);
    int block = 256, grid = nk_grid_for(ctx, p.total, block, 8);
    if (dtype == NK_F32) nk_fill_fun_kernel<float><<<grid, block, 0, ctx->stream>>>(data_of<float>(drn), p, fun, d >= 0, float(value));
    else nk_fill_fun_kernel<double><<<grid, block, 0, ctx->stream>>>(data_of<double>(drn), p, fun, d >= 0, value);
    return nk_after_launch(ctx, "nk_fill_fun_kernel");
}

template <class T>
static int sum_impl(nk_ctx* ctx, const T* in, const EwPlan& p, int64_t n, T* out_elem) {
    // levels n -> ceil(n / 128) -> ... ping-pong inside the ctx scratch block, until one CTA can do the rest
    SumView v;
    memset(&v, 0, sizeof(v));
    v.nd = p.nd;
    v.base = p.b0;
    for (int k = 0; k < p.nd; k++) { v.div[k] = p.div[k]; v.s[k] = p.s0[k]; }
    if (p.nd == 1 && p.row_major && p.s0[0] == 1) {   // contiguous
        in += p.b0;
        v.nd = 0;
        v.base = 0;
    }
    bool rows = v.nd == 0 && aligned16(in);
    T *bufA = nullptr, *bufB = nullptr;
    if (n > NK_SUM_LAST) {
        const int64_t n1 = (n + 127) / 128, n2 = (n1 + 127) / 128;
        void* scratch = nullptr;
        int st = nk_scratch(ctx, size_t(n1 + n2 + 16) * sizeof(T), &scratch);
        if (st) return st;
        bufA = reinterpret_cast<T*>(scratch);
        bufB = bufA + ((n1 + 7) / 8) * 8;   // 16-byte aligned like bufA
        NK_CUDA(ctx, cudaFuncSetAttribute(nk_sum_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, SumRows<T>::SMEM));
    }
    const T* src = in;
    int64_t cur = n;
    T* dst = bufA;
    while (cur > NK_SUM_LAST) {
        const int64_t tiles = (cur + 127) / 128;
        const char* name;
        if (rows && nk_sum_by_rows(tiles, ctx->prop.multiProcessorCount)) {
            name = "nk_sum_rows_kernel";
            using C = SumRows<T>;
            nk_sum_rows_kernel<T><<<nk_grid_for(ctx, (tiles + 31) / 32, C::WARPS, 12), C::WARPS * 32, C::SMEM, ctx->stream>>>(src, cur, dst, tiles);
        } else if (!rows && nk_sum_by_groups(tiles, v.nd, ctx->prop.multiProcessorCount)) {
            name = "nk_sum_tiles_kernel";
            if (v.nd == 0) {   // (asking for it in the kernel costs views 5 %)
                v.nd = 1;
                v.div[0] = v.s[0] = 1;
            }
            nk_sum_tiles_kernel<T><<<nk_grid_for(ctx, (tiles + 31) / 32, 4, 16), 128, 0, ctx->stream>>>(src, v, cur, dst, tiles);
        } else {
            name = "nk_sum_warp_kernel";
            nk_sum_warp_kernel<T><<<nk_grid_for(ctx, tiles, 4, 16), 128, 0, ctx->stream>>>(src, v, cur, dst, tiles);
        }
        const int st = nk_after_launch(ctx, name);
        if (st) return st;
        src = dst;
        rows = true;   // the next levels are dense
        v.nd = 0;
        v.base = 0;
        cur = tiles;
        dst = (dst == bufA) ? bufB : bufA;
    }
    nk_sum_last_kernel<T><<<1, int((cur + 127) / 128) * 32, 0, ctx->stream>>>(src, v, int(cur), out_elem);
    return nk_after_launch(ctx, "nk_sum_last_kernel");
}

extern "C" int nk_sum(nk_ctx* ctx, int32_t dtype, int32_t rank, nk_buf* src, const int32_t* cfg, nk_buf* out, int64_t out_index) {
    NK_CHECK_CTX(ctx);
    if (dtype != NK_F32 && dtype != NK_F64) return nk_fail(ctx, NK_ERR_UNSUPPORTED, "nk_sum: dtype %d not supported (F32/F64 only)", dtype);
    NkView v;
    int st;
    if ((st = nk_view_parse(ctx, "nk_sum(src)", src, cfg, rank, dtype, &v))) return st;
    if (out == nullptr || out->magic != 0x4e4b4246 || out->dtype != dtype) return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_sum: invalid output buffer");
    if (out->device != ctx->device)
        return nk_fail(ctx, NK_ERR_BAD_ARG, "nk_sum: output buffer lives on device %d, context on device %d", out->device, ctx->device);
    if (out_index < 0 || out_index >= out->n_elems) return nk_fail(ctx, NK_ERR_BOUNDS, "nk_sum: output index %lld outside the buffer", (long long)out_index);
    EwPlan p;
    make_plan(v, nullptr, nullptr, nullptr, nullptr, &p);
    if (dtype == NK_F32) return sum_impl<float>(ctx, data_of<float>(src), p, v.size, data_of<float>(out) + out_index);
    return sum_impl<double>(ctx, data_of<double>(src), p, v.size, data_of<double>(out) + out_index);
}
