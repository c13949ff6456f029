// True 32-bit matrix product  C[M,N] = A[M,K] * W[N,K]^T  (+ nothing else).
//
// The float32 path's only matrix product: 32-bit fused multiply-adds, no tensor cores, no reduced-precision mode.
//
// One order of additions, whatever M is and wherever a row sits in the batch, so that a token's result is bit-identical
// under every split of the work.  k is cut into blocks of 32.  A block's sum is that of two chains of fused multiply-adds
// from zero, one over its even and one over its odd k, both ascending (two chains because fma.rn.f32x2 runs them side by
// side on neighbouring k, which a 16-byte load brings in neighbouring registers).  The blocks are dealt out to GF_SEG runs
// of consecutive blocks; a run adds its blocks' sums ascending; C = (r0 + r1) + (r2 + r3).  Short chains also keep the
// rounding small: it grows with a chain's length, that of a sum of sums with the square root of their number.  The runs
// are what a cluster's CTAs share: 1, 2 or 4 CTAs take 4, 2 or 1 runs each and add them through distributed shared memory.
//
// Two kernels compute it.
//   rows  (few rows): bound by reading W once.  A CTA owns 32 rows of W, a lane each, and streams them through a ring
//         of 128-k stages; a warp takes one of a stage's four blocks for up to 16 rows of A.  W [151936, 1024]: 95.5 us
//         at one row (6.5 TB/s), 112 at four; from eight on (173 us) reading A from shared memory is the bound.
//   tile  (many rows): bound by the multiply-adds and their operands' way from shared memory.  64 x 64 outputs a CTA, 8 x 4 a
//         thread, three CTAs an SM: 600 x 6144 x 1024 in 209 us (36 TFLOP/s; 64 x 128 outputs, 8 x 8 a thread, two CTAs: 223).
// One kernel of 64 x 64 tiles, 4 x 4 a thread, without a ring or a split of K took 170 ms of the 207 that four prompts of
// 33 to 257 tokens and eight single tokens of each took a 28-layer model of width 1,024; the two take about 27.
//
// The reference's fp32 route is cublasSgemm (src/compute/gemm.cu:341-358) and a warp-per-row GEMV (src/compute/gemm.cu:
// 452-493); W is stored [N,K] as there (src/compute/gemm.h:18-19).
#include "common.cuh"

namespace {

constexpr int GF_BLK = 32;   // k of a block
constexpr int GF_SEG = 4;    // runs of blocks

__host__ __device__ __forceinline__ int gf_blocks(int K) { return (K + GF_BLK - 1) / GF_BLK; }
__host__ __device__ __forceinline__ int gf_run_start(int run, int n_blocks) { return (int)((int64_t)run * n_blocks / GF_SEG); }

__device__ __forceinline__ uint32_t gf_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes (four values) from global to shared memory, of which the first `valid` values are read and the rest are zero
__device__ __forceinline__ void gf_copy16(uint32_t dst, const float* src, int valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid * 4));
}
__device__ __forceinline__ void gf_copy4(uint32_t dst, const float* src, int valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid * 4));
}
__device__ __forceinline__ void gf_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void gf_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Four values at row[k ...] of a row of K values (row null: zeros) to dst.
template <bool ALIGNED>
__device__ __forceinline__ void gf_fetch(uint32_t dst, const float* row, const float* any, int k, int K) {
    if (ALIGNED) {
        const int valid = row ? max(0, min(4, K - k)) : 0;
        gf_copy16(dst, valid ? row + k : any, valid);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int valid = row && k + e < K;
            gf_copy4(dst + 4 * e, valid ? row + k + e : any, valid);
        }
    }
}

__device__ __forceinline__ void gf_fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ float gf_pair_sum(unsigned long long v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}

__device__ __forceinline__ float gf_remote(const float* p, int rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(gf_smem(p)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void gf_cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

// ------------------------------------------------------------------------------------------------ few rows
constexpr int GR_ROWS = 32;                 // rows of W of a CTA: one a lane (two halve the loads of A, and were slower: fewer CTAs an SM)
constexpr int GR_WARPS = 4;                 // a warp per block of a stage
constexpr int GR_K = GF_BLK * GR_WARPS;     // k of a stage
constexpr int GR_PITCH = GR_K + 4;          // of a row of W in shared memory: eight rows' 16-byte pieces in eight bank groups
constexpr int GR_STAGES = 3;

template <int MT> constexpr int gr_smem_floats() {
    return GR_STAGES * (GR_ROWS * GR_PITCH + MT * GR_K) + 2 * GR_WARPS * MT * GR_ROWS + GF_SEG * MT * GR_ROWS;
}

// Grid (ctas x groups of 32 rows of W, groups of MT rows of A); a cluster along x of `ctas` = 1, 2 or 4.
// early (see imp_early_weights): the first pieces of W are asked for before the kernels ahead are done.
template <int MT, bool ALIGNED>
__global__ void __launch_bounds__(GR_WARPS * 32) gemm_f32_rows_kernel(float* __restrict__ C, int64_t ldc, const float* __restrict__ A, int64_t lda,
                                                                      const float* __restrict__ W, int64_t ldw, int M, int N, int K, int ctas, int early) {
    extern __shared__ __align__(16) float gr_mem[];
    float* ws = gr_mem;                                              // [stage][GR_ROWS][GR_PITCH]
    float* as = ws + GR_STAGES * GR_ROWS * GR_PITCH;                 // [stage][MT][GR_K]
    float* part = as + GR_STAGES * MT * GR_K;                        // [2][block][MT][GR_ROWS]
    float* runs = part + 2 * GR_WARPS * MT * GR_ROWS;                // [run of this CTA][MT][GR_ROWS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % ctas, n0 = blockIdx.x / ctas * GR_ROWS, m0 = blockIdx.y * MT;
    const int n_blocks = gf_blocks(K), per = GF_SEG / ctas, run0 = rank * per;
    constexpr int OUTS = MT * GR_ROWS;

    // the stages of this CTA's runs, in order; a stage never crosses the end of a run
    struct At { int run, blk, end; };
    auto open = [&](At& s) {   // the first stage of s.run or of the next run that has one
        for (; s.run < run0 + per; ++s.run) {
            s.blk = gf_run_start(s.run, n_blocks);
            s.end = gf_run_start(s.run + 1, n_blocks);
            if (s.blk < s.end) return;
        }
    };
    auto next = [&](At& s) {
        s.blk += GR_WARPS;
        if (s.blk >= s.end) { ++s.run; open(s); }
    };
    auto fetch_w = [&](const At& s, int slot) {
        const int k0 = s.blk * GF_BLK, k1 = min(K, s.end * GF_BLK);
        constexpr int PIECES = GR_K / 4;   // a warp a row: 512 consecutive bytes
#pragma unroll
        for (int r = 0; r < GR_ROWS / GR_WARPS; ++r) {
            const int row = r * GR_WARPS + warp;
            const float* src = n0 + row < N ? W + (int64_t)(n0 + row) * ldw : nullptr;
            gf_fetch<ALIGNED>(gf_smem(ws + (slot * GR_ROWS + row) * GR_PITCH + lane * 4), src, W, k0 + lane * 4, k1);
        }
        static_assert(PIECES == 32, "a lane per piece");
    };
    auto fetch_a = [&](const At& s, int slot) {
        const int k0 = s.blk * GF_BLK, k1 = min(K, s.end * GF_BLK);
        for (int m = warp; m < MT; m += GR_WARPS) {
            const float* src = m0 + m < M ? A + (int64_t)(m0 + m) * lda : nullptr;
            gf_fetch<ALIGNED>(gf_smem(as + (slot * MT + m) * GR_K + lane * 4), src, A, k0 + lane * 4, k1);
        }
    };

    At ahead{run0, 0, 0};
    open(ahead);
    At now = ahead, first = ahead;
    if (!early) pdl_wait();
#pragma unroll
    for (int i = 0; i < GR_STAGES - 1; ++i)
        if (ahead.run < run0 + per) {
            fetch_w(ahead, i);
            next(ahead);
        }
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < GR_STAGES - 1; ++i) {
        if (first.run < run0 + per) {
            fetch_a(first, i);
            next(first);
        }
        gf_commit();   // the first of these groups holds all of W asked for above
    }
    for (int i = tid; i < per * OUTS; i += GR_WARPS * 32) runs[i] = 0.f;   // runs without a block

    constexpr int MINE = (OUTS + GR_WARPS * 32 - 1) / (GR_WARPS * 32);   // outputs whose block sums this thread adds up
    float acc[MINE];
#pragma unroll
    for (int i = 0; i < MINE; ++i) acc[i] = 0.f;
    At before{run0, 0, 0};
    bool pending = false;
    int buf = 0;
    auto add_up = [&](const At& s, const float* sums) {   // the block sums of stage s, ascending; a finished run is put away
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int o = tid + i * GR_WARPS * 32;
            if (o < OUTS) {
#pragma unroll
                for (int b = 0; b < GR_WARPS; ++b)
                    if (s.blk + b < s.end) acc[i] += sums[b * OUTS + o];
                if (s.blk + GR_WARPS >= s.end) {
                    runs[(s.run - run0) * OUTS + o] = acc[i];
                    acc[i] = 0.f;
                }
            }
        }
    };

    for (int slot = 0; now.run < run0 + per;) {
        gf_wait<GR_STAGES - 2>();
        __syncthreads();
        const int free_slot = slot == 0 ? GR_STAGES - 1 : slot - 1;   // the stage read in the round before this one
        if (ahead.run < run0 + per) {
            fetch_w(ahead, free_slot);
            fetch_a(ahead, free_slot);
            next(ahead);
        }
        gf_commit();
        if (pending) add_up(before, part + (buf ^ 1) * GR_WARPS * OUTS);
        if (now.blk + warp < now.end) {
            unsigned long long sum[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) sum[m] = 0ull;
            const float* wr = ws + (slot * GR_ROWS + lane) * GR_PITCH + warp * GF_BLK;
            const float* ar = as + slot * MT * GR_K + warp * GF_BLK;
#pragma unroll
            for (int q = 0; q < GF_BLK / 4; ++q) {
                const ulonglong2 w = *(const ulonglong2*)(wr + 4 * q);
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const ulonglong2 a = *(const ulonglong2*)(ar + m * GR_K + 4 * q);
                    gf_fma2(sum[m], a.x, w.x);
                    gf_fma2(sum[m], a.y, w.y);
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) part[(buf * GR_WARPS + warp) * OUTS + m * GR_ROWS + lane] = gf_pair_sum(sum[m]);
        }
        before = now;
        pending = true;
        buf ^= 1;
        next(now);
        slot = slot + 1 == GR_STAGES ? 0 : slot + 1;
    }
    __syncthreads();
    if (pending) add_up(before, part + (buf ^ 1) * GR_WARPS * OUTS);
    if (ctas > 1) gf_cluster_sync();
    else __syncthreads();
    for (int o = rank * (OUTS / ctas) + tid; o < (rank + 1) * (OUTS / ctas); o += GR_WARPS * 32) {
        float r[GF_SEG];
#pragma unroll
        for (int j = 0; j < GF_SEG; ++j) {
            const float* p = runs + j % per * OUTS + o;
            r[j] = j / per == rank ? *p : gf_remote(p, j / per);
        }
        const int m = m0 + o / GR_ROWS, n = n0 + o % GR_ROWS;
        if (m < M && n < N) C[(int64_t)m * ldc + n] = (r[0] + r[1]) + (r[2] + r[3]);
    }
    if (ctas > 1) gf_cluster_sync();   // nobody leaves while its sums are read
}

// ----------------------------------------------------------------------------------------------- many rows
constexpr int GT_M = 64, GT_N = 64, GT_TM = 8, GT_TN = 4, GT_THREADS = GT_M / GT_TM * (GT_N / GT_TN);
constexpr int GT_PITCH = GF_BLK + 4;
constexpr int GT_STAGES = 3;
constexpr int GT_STAGE = (GT_M + GT_N) * GT_PITCH;
constexpr int GT_OUTS = GT_M * GT_N;
constexpr int GT_SMEM = (GT_STAGES * GT_STAGE + GT_OUTS) * 4;   // the ring and one set of sums

// Grid (ctas x tiles of N, tiles of M); a cluster along x of `ctas` = 2 or 4.
template <bool ALIGNED>
__global__ void __launch_bounds__(GT_THREADS, 3) gemm_f32_tile_kernel(float* __restrict__ C, int64_t ldc, const float* __restrict__ A, int64_t lda,
                                                                      const float* __restrict__ W, int64_t ldw, int M, int N, int K, int ctas, int early) {
    extern __shared__ __align__(16) float gt_mem[];
    float* sums = gt_mem + GT_STAGES * GT_STAGE;   // [output of the thread][thread]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = blockIdx.x % ctas, n0 = blockIdx.x / ctas * GT_N, m0 = blockIdx.y * GT_M;
    // a warp covers 4 x 8 threads, so that a load of A meets four rows and a load of W eight: one pass over the banks each
    const int tm = (warp >> 1) * 4 + (lane >> 3), tn = (warp & 1) * 8 + (lane & 7);
    const int n_blocks = gf_blocks(K), per = GF_SEG / ctas, run0 = rank * per;
    const int b0 = gf_run_start(run0, n_blocks), b1 = gf_run_start(run0 + per, n_blocks);
    const int half = per == 2 ? gf_run_start(run0 + 1, n_blocks) : b1;   // where this CTA's first run ends

    auto fetch = [&](const float* X, int64_t ld, int r0, int R, float* dst, int blk) {
        constexpr int PIECES = GF_BLK / 4, AT_ONCE = GT_THREADS / PIECES;
        const int piece = tid % PIECES, k = blk * GF_BLK + piece * 4;
#pragma unroll
        for (int r = 0; r < GT_M / AT_ONCE; ++r) {
            const int row = r * AT_ONCE + tid / PIECES;
            gf_fetch<ALIGNED>(gf_smem(dst + row * GT_PITCH + piece * 4), r0 + row < R ? X + (int64_t)(r0 + row) * ld : nullptr, X, k, K);
        }
    };
    auto stage = [&](int i) { return gt_mem + i * GT_STAGE; };
    static_assert(GT_M == GT_N, "one fetch for both operands");
    if (!early) pdl_wait();
#pragma unroll
    for (int i = 0; i < GT_STAGES - 1; ++i)
        if (b0 + i < b1) fetch(W, ldw, n0, N, stage(i) + GT_M * GT_PITCH, b0 + i);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < GT_STAGES - 1; ++i) {
        if (b0 + i < b1) fetch(A, lda, m0, M, stage(i), b0 + i);
        gf_commit();
    }

    float acc[GT_TM][GT_TN];
#pragma unroll
    for (int i = 0; i < GT_TM; ++i)
#pragma unroll
        for (int j = 0; j < GT_TN; ++j) acc[i][j] = 0.f;
    if (half == b0 && per == 2)   // the first run has no block
        for (int i = 0; i < GT_TM * GT_TN; ++i) sums[i * GT_THREADS + tid] = 0.f;

    int slot = 0;
    for (int b = b0; b < b1; ++b) {
        gf_wait<GT_STAGES - 2>();
        __syncthreads();
        if (b + GT_STAGES - 1 < b1) {
            float* s = stage(slot == 0 ? GT_STAGES - 1 : slot - 1);
            fetch(A, lda, m0, M, s, b + GT_STAGES - 1);
            fetch(W, ldw, n0, N, s + GT_M * GT_PITCH, b + GT_STAGES - 1);
        }
        gf_commit();
        const float* ar = stage(slot) + tm * GT_PITCH;
        const float* wr = stage(slot) + GT_M * GT_PITCH + tn * GT_PITCH;
        unsigned long long blk[GT_TM][GT_TN];
#pragma unroll
        for (int i = 0; i < GT_TM; ++i)
#pragma unroll
            for (int j = 0; j < GT_TN; ++j) blk[i][j] = 0ull;
#pragma unroll
        for (int q = 0; q < GF_BLK / 4; ++q) {
            ulonglong2 w[GT_TN];
#pragma unroll
            for (int j = 0; j < GT_TN; ++j) w[j] = *(const ulonglong2*)(wr + j * (GT_N / GT_TN) * GT_PITCH + 4 * q);
#pragma unroll
            for (int i = 0; i < GT_TM; ++i) {
                const ulonglong2 a = *(const ulonglong2*)(ar + i * (GT_M / GT_TM) * GT_PITCH + 4 * q);
#pragma unroll
                for (int j = 0; j < GT_TN; ++j) gf_fma2(blk[i][j], a.x, w[j].x);
#pragma unroll
                for (int j = 0; j < GT_TN; ++j) gf_fma2(blk[i][j], a.y, w[j].y);
            }
        }
#pragma unroll
        for (int i = 0; i < GT_TM; ++i)
#pragma unroll
            for (int j = 0; j < GT_TN; ++j) acc[i][j] += gf_pair_sum(blk[i][j]);
        if (b + 1 == half && per == 2) {   // the first of two runs is complete
#pragma unroll
            for (int i = 0; i < GT_TM; ++i)
#pragma unroll
                for (int j = 0; j < GT_TN; ++j) {
                    sums[(i * GT_TN + j) * GT_THREADS + tid] = acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
        slot = slot + 1 == GT_STAGES ? 0 : slot + 1;
    }
#pragma unroll
    for (int i = 0; i < GT_TM; ++i)
#pragma unroll
        for (int j = 0; j < GT_TN; ++j) {
            float* s = sums + (i * GT_TN + j) * GT_THREADS + tid;
            *s = per == 2 ? *s + acc[i][j] : acc[i][j];
        }
    gf_cluster_sync();
    const int share = GT_TM * GT_TN / ctas;   // outputs a thread finishes
    for (int e = rank * share; e < (rank + 1) * share; ++e) {
        const float* p = sums + e * GT_THREADS + tid;
        float v;
        if (ctas == 2) v = gf_remote(p, 0) + gf_remote(p, 1);
        else v = (gf_remote(p, 0) + gf_remote(p, 1)) + (gf_remote(p, 2) + gf_remote(p, 3));
        const int m = m0 + e / GT_TN * (GT_M / GT_TM) + tm, n = n0 + e % GT_TN * (GT_N / GT_TN) + tn;
        if (m < M && n < N) C[(int64_t)m * ldc + n] = v;
    }
    gf_cluster_sync();
}

template <typename... KArgs, typename... Args>
cudaError_t gf_launch(void (*kernel)(KArgs...), dim3 grid, int threads, int smem, int ctas, cudaStream_t stream, Args... args) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = imp_pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

constexpr int GF_ROWS_MAX = 32;   // rows of A up to which W is streamed

template <int MT>
cudaError_t gr_launch(bool aligned, float* C, int64_t ldc, const float* A, int64_t lda, const float* W, int64_t ldw, int M, int N, int K, int early, cudaStream_t s) {
    // a CTA does all four runs where the groups alone give every SM two CTAs
    const int groups = (int)(((int64_t)N + GR_ROWS - 1) / GR_ROWS), sms = imp_sm_count();
    const int ctas = groups >= 2 * sms ? 1 : groups >= sms ? 2 : 4;
    const dim3 grid((unsigned)groups * ctas, (M + MT - 1) / MT);
    constexpr int smem = gr_smem_floats<MT>() * 4;
    if (aligned) return gf_launch(gemm_f32_rows_kernel<MT, true>, grid, GR_WARPS * 32, smem, ctas, s, C, ldc, A, lda, W, ldw, M, N, K, ctas, early);
    return gf_launch(gemm_f32_rows_kernel<MT, false>, grid, GR_WARPS * 32, smem, ctas, s, C, ldc, A, lda, W, ldw, M, N, K, ctas, early);
}

}  // namespace

IMP_API int imp_gemm_f32(float* C, int64_t ldc, const float* A, int64_t lda, const float* W, int64_t ldw, int M,
                         int N, int K, void* stream) {
    if (M == 0 || N == 0) return 0;
    IMP_CHECK_ARG(C && A && W && M > 0 && N > 0 && K > 0, "imp_gemm_f32: bad argument");
    IMP_CHECK_ARG(ldc >= N && lda >= K && ldw >= K, "imp_gemm_f32: leading dimension too small");
    const int64_t m_tiles = ((int64_t)M + GT_M - 1) / GT_M, n_tiles = ((int64_t)N + GT_N - 1) / GT_N;
    IMP_CHECK_ARG(m_tiles <= 65535, "imp_gemm_f32: M %d too large for one launch", M);
    cudaStream_t s = (cudaStream_t)stream;
    const bool aligned = (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 && lda % 4 == 0 && ldw % 4 == 0;
    const int early = imp_early_weights();
    cudaError_t e;
    if (M <= GF_ROWS_MAX) {
        e = M == 1   ? gr_launch<1>(aligned, C, ldc, A, lda, W, ldw, M, N, K, early, s)
            : M == 2 ? gr_launch<2>(aligned, C, ldc, A, lda, W, ldw, M, N, K, early, s)
            : M <= 4 ? gr_launch<4>(aligned, C, ldc, A, lda, W, ldw, M, N, K, early, s)
            : M <= 8 ? gr_launch<8>(aligned, C, ldc, A, lda, W, ldw, M, N, K, early, s)
                     : gr_launch<16>(aligned, C, ldc, A, lda, W, ldw, M, N, K, early, s);
    } else {
        // two CTAs a tile where those fill the device's slots, else four (257 rows of 1,024 x 3,072: 77 us, with two 178)
        const int ctas = m_tiles * n_tiles * 2 >= 3 * imp_sm_count() ? 2 : 4;
        const dim3 grid((unsigned)(n_tiles * ctas), (unsigned)m_tiles);
        e = aligned ? gf_launch(gemm_f32_tile_kernel<true>, grid, GT_THREADS, GT_SMEM, ctas, s, C, ldc, A, lda, W, ldw, M, N, K, ctas, early)
                    : gf_launch(gemm_f32_tile_kernel<false>, grid, GT_THREADS, GT_SMEM, ctas, s, C, ldc, A, lda, W, ldw, M, N, K, ctas, early);
    }
    if (e != cudaSuccess) {
        imp_set_error("imp_gemm_f32: %s", cudaGetErrorString(e));
        return (int)e;
    }
    IMP_RETURN_LAUNCH();
}
