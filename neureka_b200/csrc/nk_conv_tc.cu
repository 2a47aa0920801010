// Tensor-core family for F32 contraction-shaped convolution calls ([M,K,1] x [1,K,N], `Tensor.convDot`, `@`, and the two
// gradients of such calls): O[m, n] = sum_k A[m, k] * B[k, n] on the 5th-generation tensor cores with the 3xTF32 split.
// Replaces what the reference runs for these shapes on a GPU, `fast_CM_MM_MxKxN`
// (src/main/java/neureka/backend/main/operations/linear/internal/opencl/CLGEMM.java:44-92); the semantics are those of
// AbstractCPUConvolution.java:245-316 (forward) / :319-408 (deconvolution) restricted to contraction-shaped calls.
//
// 3xTF32. A TF32 operand keeps 11 significant bits, an F32 value 24. Every operand element v is split once into
// hi = tf32(v) (round to nearest) and lo = tf32(v - hi) (v - hi is exact in F32), and the product sum is evaluated as
// sum(lo_a*hi_b) + sum(hi_a*lo_b) + sum(hi_a*hi_b) with F32 accumulation in tensor memory: the dropped lo*lo term and
// the rounding of lo are below 2^-21 of |a||b| per term, inside the 1e-5 * sum|a||b| tolerance of the path.
//
// Launch sequence (one stream, one scratch block):
//   1. nk_gemm_offsets_kernel  -- only when an index group of the views has several dims (or the drain is wider than its own
//      strides tell): the groups flattened into offset tables. A matrix product's groups are one stride each: no tables;
//   2. nk_tc_split_kernel      -- gathers both operands into dense K-major arrays hi[rows][Kp] and lo[rows][Kp] (Kp = K
//      rounded up to 16, zero padded); an operand whose rows are the contiguous direction is transposed on the way, so
//      both reach the tensor cores K-major. It also clears the tickets of a k-split product;
//   3. nk_conv_tc_kernel       -- persistent, warp-specialised: one producer thread issues cp.async.bulk.tensor (TMA,
//      64-byte swizzle, no multicast, this GPU's memory only) into a ring of {A_hi, A_lo, B_hi, B_lo} panels of 16 k each;
//      one thread issues tcgen05.mma (kind::tf32, K = 8; six per stage) into one of two F32 accumulators in tensor memory
//      and hands stages back with tcgen05.commit; sixteen warps read finished accumulators with tcgen05.ld and scatter the
//      tile through the drain's strides or tables.
//
// Two shapes of step 3, chosen by estimated time (see nk_conv_tc_try):
//   * pairs of CTAs (cta_group::2), tile 256 x 256: each CTA stages 128 rows of A and 128 of B, 32 KiB per 16 k where a lone
//     CTA with a 128 x 256 tile stages 48. Six products of 128 x 256 x 8 take 768 cycles; the lone CTA moved 48 KiB in and
//     72 KiB out of its shared memory per stage in that time, more than the 128 bytes per cycle there are, the pair 32 + 48.
//     4096^3: 554 us, lone CTAs 596;
//   * lone CTAs, tile 128 x 128, for products with too few large tiles to fill the chip; where even these are too few, k is
//     split over several CTAs per tile: each warp leaves its part of the tile in scratch and takes a ticket, the warp that
//     draws the last one adds the parts in split order (nobody waits; the result does not depend on the order of arrival).
//
// Accumulation. The tensor core adds each product block into the accumulator with truncation (measured: a sum of K
// same-signed terms came out low by K/8 * 3 * 2^-25 relative, 9e-5 at K = 8192). A tile's sum over k is therefore cut
// into chunks of 128 k (48 accumulations, bias below 1.5e-6): the two accumulators alternate chunk by chunk, and the
// sixteen epilogue warps add every finished chunk into per-thread F32 running sums with ordinary round-to-nearest adds
// while the next chunk's products already run into the other accumulator. The running sums of a tile (a quarter of its
// columns per thread) go to the drain after its last chunk.
// Every mbarrier wait is bounded (nk_mbar_wait_bounded); on expiry the waiter raises the CTA's abort word and the
// host-visible status, all roles leave their loops, outstanding copies and tensor-core work are waited for (bounded),
// tensor memory is released and the kernel returns; the host then reports NK_ERR_TIMEOUT.
#include <cuda.h>

#include "nk_gemm_plan.h"
#include "nk_ptx.cuh"

int nk_tma_encode_2d_f32(const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, int box_cols, int box_rows, int swizzle,
                         CUtensorMap* out);

namespace {

constexpr int TC_BM = 128, TC_BK = 16;                        // rows of A a CTA stages, k per stage
constexpr int TC_THREADS = 576;                              // warp 0 producer, warp 1 tensor-core issue, warps 2..17 epilogue
constexpr unsigned TC_TMEM_COLS = 512;                       // all of it: two accumulators of up to 128 x 256 F32 per CTA
constexpr int TC_KC = 8;                                     // k blocks (of 16) per accumulation chunk
constexpr int TC_MAX_SPLITS = 16;

// CG: CTAs that share a tile (1 or 2); BN: columns of the tile
template <int CG, int BN>
struct TcCfg {
    static constexpr int TM = TC_BM * CG;                    // rows of the tile
    static constexpr int B_ROWS = BN / CG;                   // rows of B (columns of the tile) a CTA stages
    static constexpr int A_PART = TC_BM * TC_BK * 4;         // 8 KiB: one of A_hi / A_lo for a stage
    static constexpr int B_PART = B_ROWS * TC_BK * 4;
    static constexpr int STAGE_BYTES = 2 * A_PART + 2 * B_PART;   // 32 KiB for both shapes in use
    static constexpr int STAGES = 192 * 1024 / STAGE_BYTES;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
    static constexpr int EPI_COLS = BN / 4;                  // accumulator columns an epilogue warp owns (4 warps per lane quarter)
    // Instruction descriptor: F32 accumulate, TF32 x TF32, both operands K-major
    static constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(BN >> 3) << 17) | (uint32_t(TM >> 4) << 24);
};

// ---- split: v -> hi = tf32(v), lo = tf32(v - hi) ------------------------------------------------------------------------
__device__ __forceinline__ void tc_split(float v, float* hi, float* lo) {
    unsigned h;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
    float fh = __uint_as_float(h);
    if (!isfinite(fh)) fh = isfinite(v) ? __uint_as_float(__float_as_uint(v) & 0xffffe000u) : v;   // rounded past the largest finite value
    float r = isfinite(v) ? v - fh : 0.0f;
    unsigned l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(r));
    *hi = fh;
    *lo = __uint_as_float(l);
}

// One operand of the split: element (r, k) is src[offR(r) + offK(k)], the offsets a stride or (index groups of several dims) a table.
struct TcOperand {
    const float* src;             // the view's base
    const int64_t *offR, *offK;   // null: r * sR, k * sK
    int64_t sR, sK, R;
    int64_t tiles;                // CTAs for this operand
    int kfast;                    // consecutive k are consecutive in memory
    int vec;                      // 16-byte loads along the contiguous direction are legal (and there are no tables)
    float *hi, *lo;
};
struct TcSplit {
    TcOperand op[2];
    int64_t K, Kp;
    int* tickets;
    int n_tickets;
};
// Gathers an operand into hi / lo [R][Kp], zero for k >= K. A CTA takes 32 x 128 elements, 128 along the operand's contiguous
// direction (rows x k, or -- turned through shared memory on the way -- k x rows), four 16-byte loads per thread in flight
// and 16-byte stores; operands that 16-byte loads do not fit are read element by element. Both operands in one launch: the
// second's tiles follow the first's. Bound by memory: 12 bytes move per element.
// 4096^2 operands, two per product: 62 us (58 is the floor); two launches of 32 x 32 tiles with 4-byte accesses: 87 to 114.
__global__ void __launch_bounds__(256) nk_tc_split_kernel(const TcSplit p) {
    __shared__ float tile[32][129];
    const int which = int64_t(blockIdx.x) >= p.op[0].tiles ? 1 : 0;
    const TcOperand& o = p.op[which];
    const int64_t t = int64_t(blockIdx.x) - (which ? p.op[0].tiles : 0);
    if (p.n_tickets && blockIdx.x == 0)
        for (int i = threadIdx.x; i < p.n_tickets; i += 256) p.tickets[i] = 0;
    const int64_t tiles_k = (p.Kp + (o.kfast ? 127 : 31)) / (o.kfast ? 128 : 32);
    const int64_t k0 = (t % tiles_k) * (o.kfast ? 128 : 32), r0 = (t / tiles_k) * (o.kfast ? 32 : 128);
    auto at = [&](int64_t r, int64_t k) { return (o.offR ? o.offR[r] : r * o.sR) + (o.offK ? o.offK[k] : k * o.sK); };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float v[4][4];
    // lane: 4 consecutive elements of the contiguous direction; warp + 8 i: the other direction
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int64_t slow = (o.kfast ? r0 : k0) + warp + 8 * i, fast = (o.kfast ? k0 : r0) + lane * 4;
        const int64_t slow_end = o.kfast ? o.R : p.K, fast_end = o.kfast ? p.K : o.R;
        if (o.vec && slow < slow_end && fast + 4 <= fast_end) {
            *reinterpret_cast<float4*>(v[i]) = __ldcs(reinterpret_cast<const float4*>(o.src + (o.kfast ? at(slow, fast) : at(fast, slow))));
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) v[i][e] = slow < slow_end && fast + e < fast_end ? o.src[o.kfast ? at(slow, fast + e) : at(fast + e, slow)] : 0.0f;
        }
    }
    int64_t row[4], k;
    if (o.kfast) {
        k = k0 + lane * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) row[i] = r0 + warp + 8 * i;
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) tile[warp + 8 * i][lane * 4 + e] = v[i][e];
        __syncthreads();
        // eight lanes cover the 32 k of a row, four rows per warp and step
        k = k0 + (lane & 7) * 4;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = (lane >> 3) + 4 * (warp + 8 * i);
            row[i] = r0 + r;
#pragma unroll
            for (int e = 0; e < 4; e++) v[i][e] = tile[(lane & 7) * 4 + e][r];
        }
    }
    if (k >= p.Kp) return;   // Kp is a multiple of 16: whole vectors from here on
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (row[i] >= o.R) continue;
        float h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; e++) tc_split(v[i][e], &h[e], &l[e]);
        *reinterpret_cast<float4*>(o.hi + row[i] * p.Kp + k) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(o.lo + row[i] * p.Kp + k) = make_float4(l[0], l[1], l[2], l[3]);
    }
}

// ---- tcgen05 wrappers ------------------------------------------------------------------------------------------------
// Shared-memory operand descriptor, K-major, 64-byte swizzle: rows of 64 bytes (16 F32), 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr & 0x3ffffu) >> 4);     // start address, 16-byte units
    d |= uint64_t(1) << 16;                     // leading byte offset: not used by swizzled K-major layouts
    d |= uint64_t(512 >> 4) << 32;              // stride byte offset between 8-row groups
    d |= uint64_t(1) << 46;                     // descriptor version of this architecture
    d |= uint64_t(4) << 61;                     // layout type: 64-byte swizzle
    return d;
}
template <int CG>
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    if (CG == 2)
        asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
                     ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
                     ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// Arrives on the mbarrier (of both CTAs of a pair) once every tcgen05.mma issued so far by this thread has completed.
template <int CG>
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                     ::"r"(a), "h"((unsigned short)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(a) : "memory");
}
// the shared::cluster address of an mbarrier's counterpart in the pair's first CTA, which issues the products
__device__ __forceinline__ unsigned tc_leader_bar(uint64_t* bar) {
    unsigned a = (unsigned)__cvta_generic_to_shared(bar), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ void tc_arrive_cluster(unsigned bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// 2-D tile load of one CTA of a pair into its own shared memory, reporting to the leader's mbarrier
__device__ __forceinline__ void tc_load_pair(void* smem, const void* tensor_map, unsigned leader_bar, int c0, int c1) {
    unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    unsigned long long m = reinterpret_cast<unsigned long long>(tensor_map);
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
                 ::"r"(d), "l"(m), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
__device__ __forceinline__ void tc_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// 16 consecutive accumulator columns of this thread's lane (32 lanes x 32 bits per warp and column)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

struct TcParams {
    int64_t M, N;
    int k_blocks;                  // Kp / 16
    int tiles_m;
    int64_t units;                 // tiles * splits; unit u is part u % splits of tile u / splits
    int splits, kb_per;            // k blocks per part
    const int64_t *offOm, *offOn;  // null: m * sOm, n * sOn
    int64_t sOm, sOn, bO;
    int out_vec;                   // the drain's n index is its contiguous direction and every row starts 16-byte aligned
    float* parts;                  // splits > 1: [tile][part][warp of 16][4 columns][32 rows x 4]
    int* tickets;                  // splits > 1: [tile][warp of 16]
    int* status;                   // host-mapped word, set non-zero when a bounded wait ran out
};

template <int CG, int BN>
__global__ void __launch_bounds__(TC_THREADS, 1)
nk_conv_tc_kernel(float* __restrict__ out, const __grid_constant__ CUtensorMap mAhi, const __grid_constant__ CUtensorMap mAlo,
                  const __grid_constant__ CUtensorMap mBhi, const __grid_constant__ CUtensorMap mBlo, const __grid_constant__ TcParams p) {
    using C = TcCfg<CG, BN>;
    constexpr int STAGES = C::STAGES, EC = C::EPI_COLS;
    extern __shared__ unsigned char tc_smem_raw[];
    // stages must start on a 1024-byte boundary (swizzle pattern = function of the address bits); the dynamic block of both CTAs
    // of a pair starts at the same offset, so the pair's panels and barriers lie at the same offsets too
    unsigned char* smem = tc_smem_raw + ((1024u - ((unsigned)__cvta_generic_to_shared(tc_smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * C::STAGE_BYTES);
    uint64_t* full_bar = bars;                      // [STAGES] a stage's panels have landed (a pair's: in both CTAs; the leader's is used)
    uint64_t* empty_bar = bars + STAGES;            // [STAGES] the products reading a stage have completed
    uint64_t* acc_full = bars + 2 * STAGES;         // [2] an accumulator holds a finished chunk
    uint64_t* acc_empty = bars + 2 * STAGES + 2;    // [2] the epilogue (of both CTAs) has read it out; the leader's is used
    uint64_t* drain_bar = bars + 2 * STAGES + 4;    // only on the abort path: all issued products have completed
    volatile int* abort_word = reinterpret_cast<volatile int*>(bars + 2 * STAGES + 5);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 6);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CG == 2 ? int(blockIdx.x & 1u) : 0;              // the cluster is (2, 1, 1): rank = index inside it
    const int64_t unit0 = CG == 2 ? blockIdx.x >> 1 : blockIdx.x, unit_step = CG == 2 ? gridDim.x >> 1 : gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) { nk_mbar_init(&full_bar[s], 1); nk_mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; b++) { nk_mbar_init(&acc_full[b], 1); nk_mbar_init(&acc_empty[b], 16 * CG); }
        nk_mbar_init(drain_bar, 1);
        *abort_word = 0;
        nk_fence_barrier_init();
        nk_fence_proxy_async();
    }
    if (warp == 1) {   // one warp allocates all of the SM's tensor memory (one CTA per SM: 192 KiB of shared memory each)
        unsigned slot = (unsigned)__cvta_generic_to_shared(tmem_slot);
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(TC_TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(TC_TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();
    if (CG == 2) tc_cluster_sync();   // the peer's barriers are initialised and both allocations made
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    auto wait_or_abort = [&](uint64_t* bar, unsigned parity) -> bool {
        const int r = nk_mbar_wait_bounded(bar, parity, NK_WAIT_LIMIT_NS, abort_word);
        if (r < 0) {
            *abort_word = 1;
            if (p.status) atomicExch(p.status, 1);
        }
        return r > 0;
    };
    // the k blocks of a unit
    auto range = [&](int64_t u, int* kb_begin, int* kb_end) {
        const int part = p.splits > 1 ? int(u % p.splits) : 0;
        *kb_begin = part * p.kb_per;
        *kb_end = *kb_begin + p.kb_per < p.k_blocks ? *kb_begin + p.kb_per : p.k_blocks;
    };

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer: four tensor copies per stage; of a pair, each CTA's producer fetches its own rows ----
            int it = 0;
            bool ok = true;
            for (int64_t u = unit0; u < p.units && ok; u += unit_step) {
                const int64_t t = p.splits > 1 ? u / p.splits : u;
                int kb_begin, kb_end;
                range(u, &kb_begin, &kb_end);
                const int m0 = int(t % p.tiles_m) * C::TM + rank * TC_BM, n0 = int(t / p.tiles_m) * BN + rank * C::B_ROWS;
                for (int kb = kb_begin; kb < kb_end && ok; kb++, it++) {
                    const int s = it % STAGES;
                    ok = wait_or_abort(&empty_bar[s], ((unsigned(it) / STAGES) & 1u) ^ 1u);
                    if (!ok) break;
                    unsigned char* st = smem + size_t(s) * C::STAGE_BYTES;
                    if (rank == 0) nk_mbar_expect_tx(&full_bar[s], unsigned(CG * C::STAGE_BYTES));
                    const int k0 = kb * TC_BK;
                    if (CG == 2) {
                        const unsigned bar = tc_leader_bar(&full_bar[s]);
                        tc_load_pair(st, &mAhi, bar, k0, m0);
                        tc_load_pair(st + C::A_PART, &mAlo, bar, k0, m0);
                        tc_load_pair(st + 2 * C::A_PART, &mBhi, bar, k0, n0);
                        tc_load_pair(st + 2 * C::A_PART + C::B_PART, &mBlo, bar, k0, n0);
                    } else {
                        nk_tma_load_2d(st, &mAhi, &full_bar[s], k0, m0);
                        nk_tma_load_2d(st + C::A_PART, &mAlo, &full_bar[s], k0, m0);
                        nk_tma_load_2d(st + 2 * C::A_PART, &mBhi, &full_bar[s], k0, n0);
                        nk_tma_load_2d(st + 2 * C::A_PART + C::B_PART, &mBlo, &full_bar[s], k0, n0);
                    }
                }
            }
            if ((!ok || *abort_word) && rank == 0) {
                // copies already requested still land in shared memory: wait for them (bounded); of a pair, the leader's
                // barriers count both CTAs' bytes and neither leaves before the cluster barrier at the end
                for (int j = (it > STAGES ? it - STAGES : 0); j < it; j++)
                    nk_mbar_wait_bounded(&full_bar[j % STAGES], (unsigned(j) / STAGES) & 1u, NK_WAIT_LIMIT_NS, nullptr);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // ---- tensor-core issue: per stage two k-steps of 8, three products each (small terms first); a new
            // accumulator every TC_KC stages ----
            int it = 0, ch = 0;
            bool ok = true;
            for (int64_t u = unit0; u < p.units && ok; u += unit_step) {
                int kb_begin, kb_end;
                range(u, &kb_begin, &kb_end);
                for (int kb0 = kb_begin; kb0 < kb_end && ok; kb0 += TC_KC, ch++) {
                    const int b = ch & 1;
                    ok = wait_or_abort(&acc_empty[b], ((unsigned(ch) >> 1) & 1u) ^ 1u);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t acc = tmem_base + uint32_t(b) * BN;
                    const int kb1 = kb0 + TC_KC < kb_end ? kb0 + TC_KC : kb_end;
                    for (int kb = kb0; kb < kb1 && ok; kb++, it++) {
                        const int s = it % STAGES;
                        ok = wait_or_abort(&full_bar[s], (unsigned(it) / STAGES) & 1u);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem + size_t(s) * C::STAGE_BYTES);
#pragma unroll
                        for (int ks = 0; ks < TC_BK / 8; ks++) {
                            const uint32_t koff = uint32_t(ks) * 32u;   // 8 F32 further along the 64-byte row
                            const uint64_t a_hi = tc_smem_desc(sa + koff), a_lo = tc_smem_desc(sa + C::A_PART + koff);
                            const uint64_t b_hi = tc_smem_desc(sa + 2 * C::A_PART + koff), b_lo = tc_smem_desc(sa + 2 * C::A_PART + C::B_PART + koff);
                            tc_mma<CG>(acc, a_lo, b_hi, C::IDESC, (kb > kb0 || ks != 0) ? 1u : 0u);
                            tc_mma<CG>(acc, a_hi, b_lo, C::IDESC, 1u);
                            tc_mma<CG>(acc, a_hi, b_hi, C::IDESC, 1u);
                        }
                        tc_commit<CG>(&empty_bar[s]);   // the stage goes back to the producer(s) when these products are done
                    }
                    if (ok) tc_commit<CG>(&acc_full[b]);    // ... and the chunk to the epilogue(s)
                }
            }
            if (!ok || *abort_word) {
                tc_commit<CG>(drain_bar);           // nothing of this CTA may still run on the tensor cores at release time
                nk_mbar_wait_bounded(drain_bar, 0, NK_WAIT_LIMIT_NS, nullptr);
            }
        }
    } else {
        // ---- epilogue: warps 2..17; warp w reads the 32 accumulator lanes of its quarter (w % 4) and the columns of
        // part (w - 2) / 4, adds every finished chunk into its running sums and stores them after the tile's last chunk ----
        const int q = warp & 3, quarter = (warp - 2) >> 2;
        const unsigned empty_leader[2] = {CG == 2 ? tc_leader_bar(&acc_empty[0]) : 0u, CG == 2 ? tc_leader_bar(&acc_empty[1]) : 0u};
        int ch = 0;
        bool ok = true;
        for (int64_t u = unit0; u < p.units && ok; u += unit_step) {
            const int64_t t = p.splits > 1 ? u / p.splits : u;
            int kb_begin, kb_end;
            range(u, &kb_begin, &kb_end);
            const int64_t m = int64_t(t % p.tiles_m) * C::TM + rank * TC_BM + q * 32 + lane;
            const int64_t n0 = int64_t(t / p.tiles_m) * BN + quarter * EC;
            float sum[EC];
            for (int kb0 = kb_begin; kb0 < kb_end && ok; kb0 += TC_KC, ch++) {
                const int b = ch & 1;
                ok = wait_or_abort(&acc_full[b], (unsigned(ch) >> 1) & 1u);
                if (!ok) break;
                tc_fence_after();
                const uint32_t src = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(b) * BN + uint32_t(quarter) * EC;
#pragma unroll
                for (int c = 0; c < EC / 16; c++) {
                    uint32_t v[16];
                    tc_ld16(src + uint32_t(c) * 16u, v);
                    if (kb0 == kb_begin) {
#pragma unroll
                        for (int j = 0; j < 16; j++) sum[c * 16 + j] = __uint_as_float(v[j]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) sum[c * 16 + j] += __uint_as_float(v[j]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2) tc_arrive_cluster(empty_leader[b]);
                    else nk_mbar_arrive(&acc_empty[b]);
                }
            }
            if (!ok) continue;
            if (CG == 1 && p.splits > 1) {   // (pairs never split k)
                // this warp's part of the tile into scratch (lanes side by side), then a ticket; the last one adds all parts
                const int64_t block = int64_t(32) * EC;
                const int64_t first = ((t * p.splits) * 16 + (warp - 2)) * block;
                float4* mine = reinterpret_cast<float4*>(p.parts + first + int64_t(u % p.splits) * 16 * block);
#pragma unroll
                for (int c = 0; c < EC / 4; c++) mine[c * 32 + lane] = make_float4(sum[4 * c], sum[4 * c + 1], sum[4 * c + 2], sum[4 * c + 3]);
                __threadfence();
                __syncwarp();
                int drawn = 0;
                if (lane == 0) drawn = atomicAdd(&p.tickets[t * 16 + (warp - 2)], 1);
                drawn = __shfl_sync(0xffffffffu, drawn, 0);
                if (drawn != p.splits - 1) continue;
                __threadfence();
                for (int part = 0; part < p.splits; part++) {
                    const float4* src = reinterpret_cast<const float4*>(p.parts + first + int64_t(part) * 16 * block);
#pragma unroll
                    for (int c = 0; c < EC / 4; c++) {
                        const float4 v = __ldcg(src + c * 32 + lane);
                        if (part == 0) { sum[4 * c] = v.x; sum[4 * c + 1] = v.y; sum[4 * c + 2] = v.z; sum[4 * c + 3] = v.w; }
                        else { sum[4 * c] += v.x; sum[4 * c + 1] += v.y; sum[4 * c + 2] += v.z; sum[4 * c + 3] += v.w; }
                    }
                }
            }
            if (m >= p.M) continue;
            const int64_t row = p.bO + (p.offOm ? p.offOm[m] : m * p.sOm);
#pragma unroll
            for (int c = 0; c < EC / 32; c++) {
                const int64_t n = n0 + c * 32;
                if (n >= p.N) continue;
                if (p.out_vec && n + 32 <= p.N) {
                    float4* dst = reinterpret_cast<float4*>(out + row + n);
#pragma unroll
                    for (int j = 0; j < 8; j++) dst[j] = make_float4(sum[c * 32 + 4 * j], sum[c * 32 + 4 * j + 1], sum[c * 32 + 4 * j + 2], sum[c * 32 + 4 * j + 3]);
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (n + j < p.N) out[row + (p.offOn ? p.offOn[n + j] : (n + j) * p.sOn)] = sum[c * 32 + j];
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (CG == 2) tc_cluster_sync();   // the peer's products read this CTA's shared memory and write its tensor memory
    if (warp == 1) {
        tc_fence_after();
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TC_TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TC_TMEM_COLS) : "memory");
    }
}

template <int CG, int BN>
int tc_launch(nk_ctx* ctx, float* out, int64_t M, int64_t N, int64_t Kp, const float* Ahi, const float* Alo, const float* Bhi, const float* Blo, const TcParams& tp) {
    using C = TcCfg<CG, BN>;
    CUtensorMap mAhi, mAlo, mBhi, mBlo;
    if (nk_tma_encode_2d_f32(Ahi, uint64_t(M), uint64_t(Kp), uint64_t(Kp) * 4, TC_BK, TC_BM, 2, &mAhi) ||
        nk_tma_encode_2d_f32(Alo, uint64_t(M), uint64_t(Kp), uint64_t(Kp) * 4, TC_BK, TC_BM, 2, &mAlo) ||
        nk_tma_encode_2d_f32(Bhi, uint64_t(N), uint64_t(Kp), uint64_t(Kp) * 4, TC_BK, C::B_ROWS, 2, &mBhi) ||
        nk_tma_encode_2d_f32(Blo, uint64_t(N), uint64_t(Kp), uint64_t(Kp) * 4, TC_BK, C::B_ROWS, 2, &mBlo))
        return -1;   // no tensor-map encoder: the FMA family takes the call
    auto* kern = nk_conv_tc_kernel<CG, BN>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
    if (e != cudaSuccess) return nk_cuda_fail(ctx, e, "cudaFuncSetAttribute(nk_conv_tc_kernel)");
    const int64_t slots = ctx->prop.multiProcessorCount / CG;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(unsigned((tp.units < slots ? tp.units : slots) * CG));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = CG;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, out, mAhi, mAlo, mBhi, mBlo, tp);
    if (e != cudaSuccess) return nk_cuda_fail(ctx, e, "cudaLaunchKernelEx(nk_conv_tc_kernel)");
    return nk_after_launch(ctx, CG == 2 ? "nk_conv_tc_kernel<3xtf32,pair>" : "nk_conv_tc_kernel<3xtf32>");
}

}  // namespace

int nk_conv_tc_try(nk_ctx* ctx, nk_buf* drn, nk_buf* s1, nk_buf* s2, const GemmPlan& p, bool* handled) {
    *handled = false;
    const bool forced = ctx->conv_path == NK_CONV_TC;
    // worth three extra launches and a pass over both operands only for real matrix products
    if (p.M < 64 || p.N < 64 || p.K < 32) return NK_OK;
    if (!forced && double(p.M) * double(p.N) * double(p.K) < double(1 << 24)) return NK_OK;
    if (p.K > (int64_t(1) << 21) - 32 || p.M >= (int64_t(1) << 31) || p.N >= (int64_t(1) << 31)) return NK_OK;
    const int64_t Kp = ((p.K + TC_BK - 1) / TC_BK) * TC_BK;
    const int64_t sms = ctx->prop.multiProcessorCount;
    const int kb = int(Kp / TC_BK);
    const int64_t m_pair = (p.M + 255) / 256, n_pair = (p.N + 255) / 256, m_one = (p.M + 127) / 128, n_one = (p.N + 127) / 128;
    if (m_one * n_one > 0x7fffffffLL) return NK_OK;
    if (size_t(TcCfg<2, 256>::SMEM_BYTES) > size_t(ctx->prop.sharedMemPerBlockOptin)) return NK_OK;
    // k split of the small tiles: as many parts as keep one wave of CTAs busy, each at least two accumulation chunks long
    int splits = int(sms / (m_one * n_one));
    if (splits > kb / (2 * TC_KC)) splits = kb / (2 * TC_KC);
    if (splits > TC_MAX_SPLITS) splits = TC_MAX_SPLITS;
    if (splits < 1) splits = 1;
    const int kb_per = (kb + splits - 1) / splits;
    splits = (kb + kb_per - 1) / kb_per;
    // Estimated cycles of either shape: waves x k blocks x cycles per stage (pairs: 768, the tensor cores' time for six 128 x 256 x 8
    // products; lone CTAs: 640, their shared-memory traffic of 80 KiB per stage).
    const int64_t est_pair = ((m_pair * n_pair + sms / 2 - 1) / (sms / 2)) * kb * 768;
    const int64_t est_one = ((m_one * n_one * splits + sms - 1) / sms) * kb_per * 640;
    const bool pair = est_pair <= est_one;
    if (pair) splits = 1;
    const int64_t tiles = pair ? m_pair * n_pair : m_one * n_one;

    // scratch: [tables | A_hi | A_lo | B_hi | B_lo | parts | tickets], the arrays on 1024-byte boundaries
    const bool tables = p.m.n > 1 || p.n.n > 1 || p.k.n > 1;
    auto round = [](size_t b) { return ((b + 1023) / 1024) * 1024; };
    const size_t tab_bytes = tables ? round(size_t(2 * (p.M + p.N + p.K)) * sizeof(int64_t)) : 0;
    const size_t a_bytes = round(size_t(p.M) * Kp * 4), b_bytes = round(size_t(p.N) * Kp * 4);
    const size_t part_bytes = splits > 1 ? size_t(tiles) * splits * 128 * 128 * 4 : 0;
    const size_t ticket_bytes = splits > 1 ? size_t(tiles) * 16 * sizeof(int) : 0;
    void* scratch = nullptr;
    int st = nk_scratch(ctx, tab_bytes + 2 * a_bytes + 2 * b_bytes + part_bytes + ticket_bytes + 1024, &scratch);
    if (st) return st;
    scratch = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(scratch) + 1023) & ~uintptr_t(1023));
    int64_t* tab = reinterpret_cast<int64_t*>(scratch);
    char* base = reinterpret_cast<char*>(scratch) + tab_bytes;
    float *Ahi = reinterpret_cast<float*>(base), *Alo = reinterpret_cast<float*>(base + a_bytes);
    float *Bhi = reinterpret_cast<float*>(base + 2 * a_bytes), *Blo = reinterpret_cast<float*>(base + 2 * a_bytes + b_bytes);
    char* rest = base + 2 * a_bytes + 2 * b_bytes;

    if (tables) {
        st = nk_gemm_build_tables(ctx, p, tab);
        if (st) return st;
    }
    TcSplit sp;
    memset(&sp, 0, sizeof(sp));
    sp.K = p.K;
    sp.Kp = Kp;
    sp.tickets = reinterpret_cast<int*>(rest + part_bytes);
    sp.n_tickets = splits > 1 ? int(tiles * 16) : 0;
    auto stride = [](const GemmDims& g, bool second) { return g.n == 1 ? (second ? g.sb[0] : g.sa[0]) : 0; };   // n == 0: extent 1
    TcOperand& A = sp.op[0];
    A.src = static_cast<const float*>(s1->ptr) + p.bA;
    A.sR = stride(p.m, false); A.sK = stride(p.k, false); A.R = p.M;
    A.hi = Ahi; A.lo = Alo;
    TcOperand& B = sp.op[1];
    B.src = static_cast<const float*>(s2->ptr) + p.bB;
    B.sR = stride(p.n, false); B.sK = stride(p.k, true); B.R = p.N;
    B.hi = Bhi; B.lo = Blo;
    if (tables) {   // [offA_m | offO_m | offB_n | offO_n | offA_k | offB_k]
        A.offR = tab; A.offK = tab + 2 * p.M + 2 * p.N;
        B.offR = tab + 2 * p.M; B.offK = tab + 2 * p.M + 2 * p.N + p.K;
    }
    // is k the contiguous direction of an operand? (the innermost dim of its k group has stride 1)
    A.kfast = p.k.n > 0 && p.k.sa[p.k.n - 1] == 1;
    B.kfast = p.k.n > 0 && p.k.sb[p.k.n - 1] == 1;
    for (TcOperand* o : {&A, &B}) {
        o->tiles = o->kfast ? ((o->R + 31) / 32) * ((Kp + 127) / 128) : ((o->R + 127) / 128) * ((Kp + 31) / 32);
        const int64_t fast = o->kfast ? o->sK : o->sR, slow = o->kfast ? o->sR : o->sK;
        o->vec = !tables && fast == 1 && slow % 4 == 0 && (reinterpret_cast<uintptr_t>(o->src) % 16) == 0;
    }
    if (A.tiles + B.tiles > 0x7fffffffLL) return NK_OK;
    nk_tc_split_kernel<<<unsigned(A.tiles + B.tiles), 256, 0, ctx->stream>>>(sp);
    if ((st = nk_after_launch(ctx, "nk_tc_split_kernel"))) return st;

    TcParams tp;
    memset(&tp, 0, sizeof(tp));
    tp.M = p.M; tp.N = p.N;
    tp.k_blocks = kb;
    tp.tiles_m = int(pair ? m_pair : m_one);
    tp.units = tiles * splits;
    tp.splits = splits;
    tp.kb_per = splits > 1 ? kb_per : kb;
    if (tables) { tp.offOm = tab + p.M; tp.offOn = tab + 2 * p.M + p.N; }
    tp.sOm = stride(p.m, true);
    tp.sOn = stride(p.n, true);
    tp.bO = p.bO;
    bool vec = p.n.n == 1 && p.n.sb[0] == 1 && (p.bO % 4) == 0 && (reinterpret_cast<uintptr_t>(drn->ptr) % 16) == 0;
    for (int d = 0; d < p.m.n && vec; d++) vec = (p.m.sb[d] % 4) == 0;
    tp.out_vec = vec ? 1 : 0;
    tp.parts = reinterpret_cast<float*>(rest);
    tp.tickets = sp.tickets;
    tp.status = ctx->tma_status_dev;
    st = pair ? tc_launch<2, 256>(ctx, static_cast<float*>(drn->ptr), p.M, p.N, Kp, Ahi, Alo, Bhi, Blo, tp)
              : tc_launch<1, 128>(ctx, static_cast<float*>(drn->ptr), p.M, p.N, Kp, Ahi, Alo, Bhi, Blo, tp);
    if (st == -1) return NK_OK;
    if (st) return st;
    *handled = true;
    return NK_OK;
}
