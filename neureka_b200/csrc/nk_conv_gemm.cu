// Forward convolutions that are dense contractions: every dim is either summed away (equal extents), or belongs to
// one operand only (the other has extent 1 there). Then O[m, n] = sum_k A[m, k] * B[k, n] with m running over the dims
// only A spans, n over the dims only B spans and k over the summed dims -- `Tensor.convDot` /
// "[M,K,1] x [1,K,N]" of the reference (Tensor_Convolution_Spec.groovy:170-215, CrossDeviceSystemTest.java:95-103).
// The generic gather family computes one output per thread and re-reads both operands through L2 for each of them;
// here a CTA owns a BM x BN output tile, stages BK-deep panels of both operands in shared memory and every thread
// keeps a TM x TN block of sums in registers (8 x 8 for F32: 64 FMAs per four 128-bit shared loads).
//
// Any view works: an index space of one dim is a stride, one of several dims is flattened on the device into an offset table
// (one launch for all of them), so the panels are gathered through offA[m] + offKa[k] / offB[n] + offKb[k] and the tile is
// scattered through offOm[m] + offOn[n]. K runs with its last dim fastest, in rising order, so the result does not depend
// on scheduling.
//
// F32: plain FMAs (the large F32 products go to nk_conv_tc.cu). F64: nk_conv_dgemm_kernel below, FP64 matrix instructions.
#include "nk_gemm_plan.h"
#include "nk_launch_rules.h"

namespace {

// tables: [offA_m | offO_m] (M each), [offB_n | offO_n] (N each), [offA_k | offB_k] (K each)
__global__ void __launch_bounds__(256) nk_gemm_offsets_kernel(int64_t* __restrict__ tab, GemmPlan p) {
    const int64_t total = p.M + p.N + p.K;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x) {
        const GemmDims* g;
        int64_t idx, *t1, *t2;
        if (i < p.M) { g = &p.m; idx = i; t1 = tab; t2 = tab + p.M; }
        else if (i < p.M + p.N) { g = &p.n; idx = i - p.M; t1 = tab + 2 * p.M; t2 = tab + 2 * p.M + p.N; }
        else { g = &p.k; idx = i - p.M - p.N; t1 = tab + 2 * p.M + 2 * p.N; t2 = tab + 2 * p.M + 2 * p.N + p.K; }
        int64_t rem = idx, a = 0, b = 0;
        for (int d = g->n - 1; d >= 0; d--) {
            const int64_t q = rem % g->ext[d];
            rem /= g->ext[d];
            a += q * g->sa[d];
            b += q * g->sb[d];
        }
        t1[idx] = a;
        t2[idx] = b;
    }
}

}  // namespace

int nk_gemm_build_tables(nk_ctx* ctx, const GemmPlan& p, int64_t* tab) {
    nk_gemm_offsets_kernel<<<nk_grid_for(ctx, p.M + p.N + p.K, 256, 4), 256, 0, ctx->stream>>>(tab, p);
    return nk_after_launch(ctx, "nk_gemm_offsets_kernel");
}

namespace {

// An index space: element offset of index i through a table, or i times a stride.
struct GemmOff {
    const int64_t* tab;
    int64_t stride;
    __device__ __forceinline__ int64_t at(int64_t i) const { return tab ? tab[i] : i * stride; }
};
struct GemmView {
    GemmOff Am, Ak, Bn, Bk, Om, On;
    int64_t M, N, K, bA, bB, bO;
};
GemmView gemm_view(const GemmPlan& p, const int64_t* tab) {   // tab null: every group has at most one dim
    GemmView v;
    auto off = [&](const GemmDims& g, bool second, int64_t at) { return GemmOff{tab ? tab + at : nullptr, g.n == 1 ? (second ? g.sb[0] : g.sa[0]) : 0}; };
    v.Am = off(p.m, false, 0);
    v.Om = off(p.m, true, p.M);
    v.Bn = off(p.n, false, 2 * p.M);
    v.On = off(p.n, true, 2 * p.M + p.N);
    v.Ak = off(p.k, false, 2 * p.M + 2 * p.N);
    v.Bk = off(p.k, true, 2 * p.M + 2 * p.N + p.K);
    v.M = p.M; v.N = p.N; v.K = p.K;
    v.bA = p.bA; v.bB = p.bB; v.bO = p.bO;
    return v;
}

// 128 x 128: 64 FMAs per four 128-bit shared loads. 64 x 64: four times the CTAs for products with less than one large tile per SM.
struct GemmTile128 { static constexpr int BM = 128, BN = 128, BK = 16, TM = 8, TN = 8; };
struct GemmTile64 { static constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4; };

// 256 threads as 16 x 16; thread (ty, tx) owns rows {ty*TM/2 .. +TM/2} of each half of the tile's rows and columns
// {tx*TN/2 .. +TN/2} of each half of its columns, so that the lanes of a quarter warp read consecutive 16-byte words.
// OFF: type the per-thread gather offsets are kept in -- 32 bits when both operands are smaller than 2^31 elements (half the
// registers of the 64-bit form, which spilled inside the main loop).
template <class T, class C, class OFF>
__global__ void __launch_bounds__(256, 2) nk_conv_gemm_kernel(T* __restrict__ out, const T* __restrict__ A, const T* __restrict__ B, const GemmView p) {
    constexpr int BM = C::BM, BN = C::BN, BK = C::BK, TM = C::TM, TN = C::TN, HM = TM / 2, HN = TN / 2;
    constexpr int PADM = BM + 4, PADN = BN + 4;
    constexpr int LA = BM * BK / 256, LB = BN * BK / 256;   // elements a thread fetches per panel
    __shared__ __align__(16) T As[2][BK][PADM];
    __shared__ __align__(16) T Bs[2][BK][PADN];

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t tilesN = (p.N + BN - 1) / BN;
    const int64_t m0 = (blockIdx.x / tilesN) * BM, n0 = (blockIdx.x % tilesN) * BN;

    // panel fetch pattern: A by (m = tid / BK + i * (256 / BK), k = tid % BK) -- k fastest, contiguous for row-major A;
    //                      B by (k = tid / BN + i * (256 / BN), n = tid % BN) -- n fastest, contiguous for row-major B
    const int ak = tid % BK, am = tid / BK;
    const int bn = tid % BN, bk = tid / BN;
    // rows / columns past the edge are clamped to the last valid one (their products land in accumulators that are
    // never stored), so the panel loads need no per-element predicate; only the K tail is guarded
    OFF a_off[LA], b_off;
#pragma unroll
    for (int i = 0; i < LA; i++) {
        int64_t m = m0 + am + i * (256 / BK);
        if (m >= p.M) m = p.M - 1;
        a_off[i] = OFF(p.bA + p.Am.at(m));
    }
    {
        int64_t n = n0 + bn;
        if (n >= p.N) n = p.N - 1;
        b_off = OFF(p.bB + p.Bn.at(n));
    }

    T ra[LA], rb[LB];
    auto fetch = [&](int64_t k0) {
        if (k0 + BK <= p.K) {
            const OFF oka = OFF(p.Ak.at(k0 + ak));
#pragma unroll
            for (int i = 0; i < LA; i++) ra[i] = A[a_off[i] + oka];
#pragma unroll
            for (int i = 0; i < LB; i++) rb[i] = B[b_off + OFF(p.Bk.at(k0 + bk + i * (256 / BN)))];
        } else {
            const int64_t ka = k0 + ak;
#pragma unroll
            for (int i = 0; i < LA; i++) ra[i] = ka < p.K ? A[a_off[i] + OFF(p.Ak.at(ka))] : T(0);
#pragma unroll
            for (int i = 0; i < LB; i++) {
                const int64_t kb = k0 + bk + i * (256 / BN);
                rb[i] = kb < p.K ? B[b_off + OFF(p.Bk.at(kb))] : T(0);
            }
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int i = 0; i < LA; i++) As[buf][ak][am + i * (256 / BK)] = ra[i];
#pragma unroll
        for (int i = 0; i < LB; i++) Bs[buf][bk + i * (256 / BN)][bn] = rb[i];
    };

    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = T(0);

    fetch(0);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int64_t k0 = 0; k0 < p.K; k0 += BK) {
        const bool more = k0 + BK < p.K;
        if (more) fetch(k0 + BK);   // global loads of the next panels fly while this one is consumed
#pragma unroll
        for (int k = 0; k < BK; k++) {
            T a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < HM; i++) { a[i] = As[buf][k][ty * HM + i]; a[HM + i] = As[buf][k][BM / 2 + ty * HM + i]; }
#pragma unroll
            for (int j = 0; j < HN; j++) { b[j] = Bs[buf][k][tx * HN + j]; b[HN + j] = Bs[buf][k][BN / 2 + tx * HN + j]; }
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (more) {
            stash(buf ^ 1);   // the other buffer was last read one iteration ago, before the barrier below
            __syncthreads();
            buf ^= 1;
        }
    }

#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int64_t m = m0 + (i < HM ? ty * HM + i : BM / 2 + ty * HM + (i - HM));
        if (m >= p.M) continue;
        const int64_t om = p.bO + p.Om.at(m);
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int64_t n = n0 + (j < HN ? tx * HN + j : BN / 2 + tx * HN + (j - HN));
            if (n < p.N) out[om + p.On.at(n)] = acc[i][j];
        }
    }
}

// ---- F64 on the FP64 matrix instructions ------------------------------------------------------------------------------
// mma.m8n8k4 multiplies an 8 x 4 by a 4 x 8 block: 256 FMAs for two 64-bit shared loads, where the FMA form spent a shared load
// on every eight. A CTA of four warps takes a 64 x 64 tile, a warp 32 x 32 of it (16 blocks, 64 accumulator registers); panels of
// 16 k lie k fastest in shared memory with a pitch of 20 doubles, which puts the 4 x 4 (row, k) elements of a half warp's
// fragment load on 16 different banks. The next panel travels through registers while this one is multiplied.
// Where the tiles are few or fill the last wave badly, k is split over several CTAs per tile (nk_dgemm_parts); every warp leaves its part in
// scratch and draws a ticket, and the one with the last ticket adds the parts in split order (nobody waits, same bits always).
constexpr int DG_T = 64, DG_K = 16, DG_PITCH = 20;
static_assert(DG_T * DG_T * sizeof(double) == NK_DGEMM_PART_BYTES, "a part is one tile of sums");
struct DgemmSplit {
    int splits, kb_per;           // k blocks of DG_K per part
    double* parts;                // [tile][part][warp of 4][16 blocks][32 lanes x 2]
    int* tickets;                 // [tile][warp of 4]
    int a_kfast, b_kfast;         // k is the operand's contiguous direction
};
__device__ __forceinline__ void dg_mma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
// TABLES: some index group goes through an offset table. Otherwise an element's address is one base per operand and thread plus
// a constant step, moved on by a panel at a time: with the offsets worked out per element, the integer chains took longer than
// the products (777 x 1023 x 515: 60 us, with offsets per element 79; 128 x 64 tiles of multiply-adds: 172). Through tables, 1024^3 in
// groups of 32 x 32: 121 us, both offsets looked up per element 168.
template <bool TABLES>
__global__ void __launch_bounds__(128, 3) nk_conv_dgemm_kernel(double* __restrict__ out, const double* __restrict__ A, const double* __restrict__ B,
                                                               const GemmView p, const DgemmSplit sp) {
    __shared__ double As[2][DG_T][DG_PITCH], Bs[2][DG_T][DG_PITCH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t tilesN = (p.N + DG_T - 1) / DG_T;
    const int part = int(blockIdx.x % unsigned(sp.splits));
    const int64_t t = blockIdx.x / unsigned(sp.splits);
    const int64_t m0 = (t / tilesN) * DG_T, n0 = (t % tilesN) * DG_T;
    const int64_t k_begin = int64_t(part) * sp.kb_per * DG_K;
    int64_t k_end = k_begin + int64_t(sp.kb_per) * DG_K;
    if (k_end > p.K) k_end = p.K;
    // element i (of 8) of a thread's share of a panel: (row, k) with the operand's contiguous direction across the threads
    auto place = [&](int kfast, int i, int* r, int* k) {
        if (kfast) { *k = tid & 15; *r = (tid >> 4) + 8 * i; }
        else { *r = tid & 63; *k = (tid >> 6) + 2 * i; }
    };
    double ra[8], rb[8];
    // rows past the edge and the k tail read as zero
    struct Walk { const double* at; int64_t step, panel; unsigned rows; int k; };   // rows: bit i = element i's row exists
    auto walk = [&](const double* base, const GemmOff& R, const GemmOff& K, int64_t row0, int64_t n_rows, int kfast) {
        Walk w;
        int r0, r;
        place(kfast, 0, &r0, &w.k);
        w.at = base + (row0 + r0) * R.stride + (k_begin + w.k) * K.stride;
        w.step = kfast ? 8 * R.stride : 2 * K.stride;
        w.panel = DG_K * K.stride;
        w.rows = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            int k;
            place(kfast, i, &r, &k);
            if (row0 + r < n_rows) w.rows |= 1u << i;
        }
        return w;
    };
    Walk wa = walk(A + p.bA, p.Am, p.Ak, m0, p.M, sp.a_kfast), wb = walk(B + p.bB, p.Bn, p.Bk, n0, p.N, sp.b_kfast);
    auto pull = [&](Walk& w, int kfast, int left, double (&v)[8]) {   // left: k of the panel that exist
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = kfast ? w.k : w.k + 2 * i;
            v[i] = ((w.rows >> i) & 1u) && k < left ? w.at[i * w.step] : 0.0;
        }
        w.at += w.panel;
    };
    // through tables: the rows' offsets are looked up once per tile, a panel's k offsets once per thread (k fastest) or element
    __shared__ int64_t row_a[TABLES ? DG_T : 1], row_b[TABLES ? DG_T : 1];
    if constexpr (TABLES) {
        if (tid < DG_T) row_a[tid] = m0 + tid < p.M ? p.bA + p.Am.at(m0 + tid) : 0;
        else row_b[tid - DG_T] = n0 + tid - DG_T < p.N ? p.bB + p.Bn.at(n0 + tid - DG_T) : 0;
        __syncthreads();
    }
    auto gather = [&](const double* base, const int64_t* rows, const GemmOff& K, int64_t row0, int64_t n_rows, int kfast, int64_t k0, double (&v)[8]) {
        int r, k;
        place(kfast, 0, &r, &k);
        if (kfast) {
            const bool ok = k0 + k < k_end;
            const int64_t ko = ok ? K.at(k0 + k) : 0;
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = ok && row0 + r + 8 * i < n_rows ? base[rows[r + 8 * i] + ko] : 0.0;
        } else {
            const bool ok = row0 + r < n_rows;
            const int64_t ro = rows[r];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = ok && k0 + k + 2 * i < k_end ? base[ro + K.at(k0 + k + 2 * i)] : 0.0;
        }
    };
    auto fetch = [&](int64_t k0) {
        if constexpr (!TABLES) {
            const int left = k_end - k0 < DG_K ? int(k_end - k0) : DG_K;
            pull(wa, sp.a_kfast, left, ra);
            pull(wb, sp.b_kfast, left, rb);
        } else {
            gather(A, row_a, p.Ak, m0, p.M, sp.a_kfast, k0, ra);
            gather(B, row_b, p.Bk, n0, p.N, sp.b_kfast, k0, rb);
        }
    };
    auto stash = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
            int r, k;
            place(sp.a_kfast, i, &r, &k);
            As[buf][r][k] = ra[i];
            place(sp.b_kfast, i, &r, &k);
            Bs[buf][r][k] = rb[i];
        }
    };
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32, fr = lane >> 2, fk = lane & 3;
    fetch(k_begin);
    stash(0);
    __syncthreads();
    int buf = 0;
    for (int64_t k0 = k_begin; k0 < k_end; k0 += DG_K) {
        const bool more = k0 + DG_K < k_end;
        if (more) fetch(k0 + DG_K);
#pragma unroll
        for (int k = 0; k < DG_K; k += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = As[buf][wm + 8 * i + fr][k + fk];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = Bs[buf][wn + 8 * j + fr][k + fk];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) dg_mma(acc[i][j], a[i], b[j]);
        }
        if (more) {
            stash(buf ^ 1);   // the other buffer was last read one panel ago, before the barrier below
            __syncthreads();
            buf ^= 1;
        }
    }
    if (sp.splits > 1) {
        const int64_t block = 16 * 64;
        const int64_t first = (t * sp.splits * 4 + warp) * block;
        double2* mine = reinterpret_cast<double2*>(sp.parts + first + int64_t(part) * 4 * block);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) mine[(i * 4 + j) * 32 + lane] = make_double2(acc[i][j][0], acc[i][j][1]);
        __threadfence();
        __syncwarp();
        int drawn = 0;
        if (lane == 0) drawn = atomicAdd(&sp.tickets[t * 4 + warp], 1);
        drawn = __shfl_sync(0xffffffffu, drawn, 0);
        if (drawn != sp.splits - 1) return;
        __threadfence();
        for (int q = 0; q < sp.splits; q++) {
            const double2* src = reinterpret_cast<const double2*>(sp.parts + first + int64_t(q) * 4 * block);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const double2 v = __ldcg(src + (i * 4 + j) * 32 + lane);
                    acc[i][j][0] = q == 0 ? v.x : acc[i][j][0] + v.x;
                    acc[i][j][1] = q == 0 ? v.y : acc[i][j][1] + v.y;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int64_t m = m0 + wm + 8 * i + fr;
        if (m >= p.M) continue;
        const int64_t om = p.bO + p.Om.at(m);
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int64_t n = n0 + wn + 8 * j + 2 * fk + e;
                if (n < p.N) out[om + p.On.at(n)] = acc[i][j][e];
            }
    }
}

// the offset tables, where a group has several dims: `extra` more bytes follow them in the scratch block
int gemm_scratch(nk_ctx* ctx, const GemmPlan& p, size_t extra, const int64_t** tab, void** rest) {
    const bool tables = p.m.n > 1 || p.n.n > 1 || p.k.n > 1;
    const size_t bytes = tables ? ((size_t(2 * (p.M + p.N + p.K)) * sizeof(int64_t) + 255) / 256) * 256 : 0;
    *tab = nullptr;
    *rest = nullptr;
    if (bytes + extra == 0) return NK_OK;
    void* scratch = nullptr;
    const int st = nk_scratch(ctx, bytes + extra, &scratch);
    if (st) return st;
    *rest = static_cast<char*>(scratch) + bytes;
    if (!tables) return NK_OK;
    *tab = static_cast<int64_t*>(scratch);
    return nk_gemm_build_tables(ctx, p, static_cast<int64_t*>(scratch));
}

template <class T, class C>
int launch_gemm_tile(nk_ctx* ctx, T* out, const T* A, const T* B, const GemmView& v, bool narrow) {
    const int64_t tiles = ((v.M + C::BM - 1) / C::BM) * ((v.N + C::BN - 1) / C::BN);
    if (tiles > 0x7fffffffLL) return -1;
    if (narrow) nk_conv_gemm_kernel<T, C, unsigned><<<unsigned(tiles), 256, 0, ctx->stream>>>(out, A, B, v);
    else nk_conv_gemm_kernel<T, C, int64_t><<<unsigned(tiles), 256, 0, ctx->stream>>>(out, A, B, v);
    return nk_after_launch(ctx, "nk_conv_gemm_kernel");
}

int launch_gemm(nk_ctx* ctx, float* out, const float* A, const float* B, const GemmPlan& p, bool narrow) {
    const int64_t* tab;
    void* rest;
    const int st = gemm_scratch(ctx, p, 0, &tab, &rest);
    if (st) return st;
    const GemmView v = gemm_view(p, tab);
    const int64_t large = ((p.M + 127) / 128) * ((p.N + 127) / 128);
    if (large < ctx->prop.multiProcessorCount) return launch_gemm_tile<float, GemmTile64>(ctx, out, A, B, v, narrow);
    return launch_gemm_tile<float, GemmTile128>(ctx, out, A, B, v, narrow);
}

int launch_gemm(nk_ctx* ctx, double* out, const double* A, const double* B, const GemmPlan& p, bool) {
    const int64_t sms = ctx->prop.multiProcessorCount;
    const int64_t tiles = ((p.M + DG_T - 1) / DG_T) * ((p.N + DG_T - 1) / DG_T);
    if (tiles > 0x3ffffffLL) return -1;
    const int64_t kb = (p.K + DG_K - 1) / DG_K;
    NkDgemmParts parts = nk_dgemm_parts(tiles, kb, sms);
    DgemmSplit sp;
    memset(&sp, 0, sizeof(sp));
    sp.a_kfast = p.k.n > 0 && p.k.sa[p.k.n - 1] == 1;
    sp.b_kfast = p.k.n > 0 && p.k.sb[p.k.n - 1] == 1;
    const int64_t* tab;
    void* rest;
    auto part_bytes = [&] { return parts.splits > 1 ? size_t(tiles) * parts.splits * NK_DGEMM_PART_BYTES : 0; };
    auto ticket_bytes = [&] { return parts.splits > 1 ? size_t(tiles) * 4 * sizeof(int) : 0; };
    int st = gemm_scratch(ctx, p, part_bytes() + ticket_bytes(), &tab, &rest);
    if (st == NK_ERR_OOM && parts.splits > 1) {   // the parts are only there for speed
        parts = NkDgemmParts{1, kb};
        st = gemm_scratch(ctx, p, 0, &tab, &rest);
    }
    if (st) return st;
    sp.splits = parts.splits;
    sp.kb_per = int(parts.kb_per);
    if (sp.splits > 1) {
        sp.parts = static_cast<double*>(rest);
        sp.tickets = reinterpret_cast<int*>(static_cast<char*>(rest) + part_bytes());
        NK_CUDA(ctx, cudaMemsetAsync(sp.tickets, 0, ticket_bytes(), ctx->stream));
    }
    if (tab) nk_conv_dgemm_kernel<true><<<unsigned(tiles * sp.splits), 128, 0, ctx->stream>>>(out, A, B, gemm_view(p, tab), sp);
    else nk_conv_dgemm_kernel<false><<<unsigned(tiles * sp.splits), 128, 0, ctx->stream>>>(out, A, B, gemm_view(p, tab), sp);
    return nk_after_launch(ctx, "nk_conv_gemm_kernel");
}

}  // namespace

// Forward calls and deconvolutions. *handled is set when the call was a contraction and has been launched.
int nk_conv_gemm_try(nk_ctx* ctx, int dtype, nk_buf* drn, const NkView& v0, nk_buf* s1, const NkView& v1, nk_buf* s2, const NkView& v2,
                     int d, bool* handled) {
    *handled = false;
    GemmPlan p;
    if (!nk_gemm_classify(v0, v1, v2, d, &p)) return NK_OK;
    // small or skinny problems stay on the gather family (one launch, no tables; a 128-wide tile would be mostly empty)
    const bool forced = ctx->conv_path != NK_CONV_AUTO;   // a forced family skips the "is it worth it" volume test only
    if (p.M < 32 || p.N < 32 || p.K < 16) return NK_OK;
    if (!forced && double(p.M) * double(p.N) * double(p.K) < double(1 << 21)) return NK_OK;
    int st;
    if (dtype == NK_F32 && ctx->conv_path != NK_CONV_GEMM) {   // the tensor-core family first; it declines what it cannot take
        st = nk_conv_tc_try(ctx, drn, s1, s2, p, handled);
        if (st) return st;
        if (*handled) { ctx->last_conv_path = NK_CONV_TC; return NK_OK; }
    }
    if (ctx->conv_path == NK_CONV_TC) return NK_OK;
    const bool narrow = s1->n_elems < (int64_t(1) << 31) && s2->n_elems < (int64_t(1) << 31);   // every gather offset fits 32 bits
    if (dtype == NK_F32) st = launch_gemm(ctx, (float*)drn->ptr, (const float*)s1->ptr, (const float*)s2->ptr, p, narrow);
    else st = launch_gemm(ctx, (double*)drn->ptr, (const double*)s1->ptr, (const double*)s2->ptr, p, narrow);
    if (st == -1) return NK_OK;
    if (st) return st;
    ctx->last_conv_path = NK_CONV_GEMM;
    *handled = true;
    return NK_OK;
}
