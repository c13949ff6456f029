// A whole stack of pre-norm decoder layers (norm, grouped-query attention over the paged cache, norm, gated feed-forward)
// for a step of up to eight single tokens, in one cooperative launch.
//
// What bounds it: every weight is read once per step, so the floor is the memory's rate (8B shape: 386 MB a layer, 59 us at
// 6.54 TB/s).  As seven launches a layer the step ran at 0.57 of that rate with one token: each launch fills and drains its own
// pipeline, and between two dependent launches the memory idles.  Here one CTA an SM lives through all layers.  A producer warp
// streams this CTA's share of every matrix (and the cached keys and values it will need) through one ring of shared memory,
// in the order in which they will be used, and never waits for the other CTAs: what it fetches does not depend on this step's
// activations.  So while the eight consumer warps wait at a grid barrier between two phases, up to 190 KB an SM (28 MB on
// the device, 4 us of the memory's time) are already on their way.
//
// Phases of a layer, a grid barrier behind each:
//   1  x = rmsnorm(h); q,k,v = x Wqkv^T          3  h += attn Wo^T         5  h += hid Wdown^T
//   2  attention of the new tokens               4  x = rmsnorm(h); hid = act(x Wgate^T) * (x Wup^T)
// A CTA owns a contiguous share of each product's output columns, to one column (4,096 columns on 148 CTAs: 27 or 28), and the
// whole contraction of it: no partial results leave the CTA.  A stage of the ring holds 8 rows of W by 1,024 of the
// contraction; each of the eight warps multiplies its own 128 of them (mma.sync m16n8k16: rows of W are the M side, two
// stages a tile, tokens the N side; the tensor rate does not matter at these shapes), with its part of x in registers.  The
// eight sums of an output meet in shared memory, in warp order.  The owner of a column of the stream adds the branch
// (rounded to bfloat16 as the other kernels store it) and leaves its share of the row's sum of squares, from which everybody
// has the norm after the barrier.
// Attention: the keys of a (sequence, kv head) are cut into as many parts as there are CTAs to take them (parts of at least
// 128 keys); a warp takes 32 keys at a time; parts merge through global memory in the CTA that comes last, in part order.
// The warp with the token's own position makes the new key (norm, rotation) and writes key and value to their page.
//
// Every wait is bounded: one that runs out reports IMP_WAIT_TIMEOUT and marks the CTA, which then runs through its
// remaining phases without waiting; the producer stops and waits (bounded) for its copies in flight.
#include "tc_common.cuh"
#include "decode_stack.h"

namespace {

constexpr int DH = 128;                       // head size
constexpr int CW = 8;                         // consumer warps
constexpr int CT = CW * 32;                   // consumer threads
constexpr int THREADS = CT + 128;             // and a warpgroup of which one warp is the producer
constexpr int KW = 128;                       // of the contraction a warp and stage
constexpr int KC = KW * CW;                   // of the contraction in a stage
constexpr int ROWS = 8;                       // rows of W in a stage
constexpr int ROW_BYTES = KC * 2;
constexpr int STAGE_BYTES = ROWS * ROW_BYTES;
constexpr int TILE = 2 * ROWS;                // rows of W in a product's tile: two stages
constexpr int BATCH = 4;                      // tiles whose sums meet at once
constexpr int SLOTS = CT / (TILE * 8);        // of them at a time: a thread an output
constexpr int TILES = 3;                      // most tiles of a CTA's share of the stream's columns
constexpr int BX = 3;                         // parts of the contraction whose x is on its way
constexpr int UNIT = 32;                      // keys in a stage
constexpr int RUN_BYTES = 16 * DH * 2;        // 16 keys lie in one page
constexpr int MIN_UNITS = 4;                  // of a part of the keys
constexpr int MAX_T = STACK_MAX_TOKENS;
constexpr int MAX_STAGES = 16;
static_assert(2 * UNIT * DH * 2 <= STAGE_BYTES, "a stage holds 32 keys and values");

struct Shared {
    uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    volatile int dead;                        // a wait ran out
    int last;                                 // this CTA's part of the keys came last
    int pos[MAX_T], seq[MAX_T];
    int units[MAX_T], parts[MAX_T], item0[MAX_T + 1];   // per token: blocks of 32 keys, parts, first item
    float ss[CW][MAX_T], inv[MAX_T];
    float m[CW][8], l[CW][8];                 // attention: per warp and query head
    alignas(16) uint32_t own_k[DH / 2];       // the token's own key and value
    alignas(16) uint32_t own_v[DH / 2];
};
constexpr int SHARED_BYTES = (sizeof(Shared) + 127) / 128 * 128;
extern __shared__ __align__(128) unsigned char stack_smem[];    // Shared | layers | scratch | ring

__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, Shared& sh, int* status) {
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if (sh.dead) return false;
    }
    sh.dead = 1;
    imp_report(status, IMP_WAIT_TIMEOUT);
    return false;
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CT) : "memory"); }

// Position in the ring, the same walk on both sides.
struct Ring {
    int slot = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next(int n) {
        if (++slot == n) slot = 0, phase ^= 1u;
    }
};

// c[16 x 8] += a[16 x 16] b[16 x 8]: rows g and g + 8 (a0 a2 and a1 a3) on the left, column g on the right; c[0], c[1]: row g, columns 2t and
// 2t + 1; c[2], c[3]: row g + 8.
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transposed(uint32_t v) {   // an 8 x 8 matrix of 16-bit values, two of a row a lane
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack(uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); }
__device__ __forceinline__ float exp2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ int share(int n, int cta, int ctas) { return (int)((int64_t)n * cta / ctas); }

// This step's items of attention: item = part of the keys of one (token, kv head).
struct Item {
    int tok, kvh, part, parts, unit0, unit1;
};
__device__ __forceinline__ Item item_of(const Shared& sh, int item, int T) {
    Item r;
    r.tok = 0;
    while (r.tok + 1 < T && item >= sh.item0[r.tok + 1]) ++r.tok;
    const int i = item - sh.item0[r.tok], n = sh.units[r.tok];
    r.parts = sh.parts[r.tok];
    r.kvh = i / r.parts;
    r.part = i - r.kvh * r.parts;
    r.unit0 = (int)((int64_t)n * r.part / r.parts);
    r.unit1 = (int)((int64_t)n * (r.part + 1) / r.parts);
    return r;
}

// ------------------------------------------------------------------------------------------------- producer
struct Producer {
    const StackArgs& a;
    Shared& sh;
    uint32_t ring, full, empty;
    int lane;
    Ring at;
    int issued = 0;
    bool ok = true;

    __device__ __forceinline__ bool slot_free() {
        if (!ok) return false;
        bool got = true;
        if (lane == 0) got = wait_bar(empty + 8 * at.slot, at.phase ^ 1u, sh, a.status);
        ok = __shfl_sync(0xffffffffu, (int)got, 0) != 0;
        return ok;
    }
    // The first eight lanes' copies make up a stage.
    __device__ __forceinline__ void issue(uint32_t dst, const void* src, uint32_t bytes) {
        uint32_t total = bytes;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0) mbar_expect_tx(full + 8 * at.slot, total);
        __syncwarp();
        if (bytes)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                         "r"(full + 8 * at.slot) : "memory");
        at.next(a.n_stages);
        ++issued;
    }
    // The lane's row of W (negative: none), part `chunk` of the contraction.
    __device__ __forceinline__ void rows(const __nv_bfloat16* w, int row, int K, int chunk) {
        if (!slot_free()) return;
        const int k = chunk * KC, n = min(KC, K - k);
        issue(ring + at.slot * STAGE_BYTES + (lane & 7) * ROW_BYTES, w + (int64_t)row * K + k, lane < 8 && row >= 0 ? (uint32_t)n * 2 : 0u);
    }
    // A product whose x stays in registers: all of the contraction for a tile of rows, then the next tile.  A tile is two stages a part
    // of the contraction: eight rows and eight more, or (gated) eight gate rows and their up rows; the last tile may want the first only.
    __device__ __forceinline__ void by_tile(const __nv_bfloat16* w, int r0, int r1, int K, bool gated) {
        const int chunks = (K + KC - 1) / KC, l = lane & 7;
        for (int r = r0; r < r1; r += gated ? ROWS : TILE)
            for (int c = 0; c < chunks; ++c) {
                if (gated) {   // gate and up rows alternate in runs of 8
                    const int row = r + l < r1 ? (r + l) / 8 * 16 + (r + l) % 8 : -1;
                    rows(w, row, K, c);
                    rows(w, row < 0 ? -1 : row + 8, K, c);
                } else {
                    rows(w, r + l < r1 ? r + l : -1, K, c);
                    if (r + ROWS < r1) rows(w, r + ROWS + l < r1 ? r + ROWS + l : -1, K, c);
                }
            }
    }
    // All tiles for a part of the contraction, then the next part.
    __device__ __forceinline__ void by_chunk(const __nv_bfloat16* w, int r0, int r1, int K) {
        const int chunks = (K + KC - 1) / KC;
        for (int c = 0; c < chunks; ++c)
            for (int r = r0; r < r1; r += ROWS) rows(w, r + (lane & 7) < r1 ? r + (lane & 7) : -1, K, c);
    }
    // Keys and values of this CTA's items.  A lane looks up the page of one run of 16 keys for sixteen blocks of 32 at once.
    __device__ __forceinline__ void keys(const StackLayer& L) {
        const int n_items = sh.item0[a.T];
        for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
            const Item it = item_of(sh, item, a.T);
            const int pos = sh.pos[it.tok];
            const int* bt = a.block_table + (int64_t)sh.seq[it.tok] * a.bt_stride;
            for (int u0 = it.unit0; u0 < it.unit1; u0 += 16) {
                const int j_lane = u0 * UNIT + lane * 16;
                const int page_lane = j_lane <= pos && u0 + (lane >> 1) < it.unit1 ? bt[j_lane / a.page_size] : -1;
                for (int u = u0; u < min(u0 + 16, it.unit1); ++u) {
                    const int run = lane & 1;
                    const int j = u * UNIT + run * 16;
                    const int page = __shfl_sync(0xffffffffu, page_lane, (u - u0) * 2 + run);
                    const bool wanted = j <= pos, good = wanted && page >= 0 && page < a.num_pages;
                    if (wanted && !good && lane < 2) imp_report(a.status, IMP_BAD_PAGE);
                    if (!slot_free()) return;
                    const int64_t off = (((int64_t)page * a.hkv + it.kvh) * a.page_size + j % a.page_size) * DH;
                    const bool value = lane & 2;
                    issue(ring + at.slot * STAGE_BYTES + (value ? 2 * RUN_BYTES : 0) + run * RUN_BYTES,
                          (const __nv_bfloat16*)(value ? L.v_pages : L.k_pages) + off, lane < 4 && good ? (uint32_t)RUN_BYTES : 0u);
                }
            }
        }
    }
    __device__ __forceinline__ void drain() {   // the copies in flight land before the memory is given back
        if (ok || lane != 0) return;
        for (int i = 0; i < min(issued, a.n_stages); ++i) {
            if (at.slot == 0) at.phase ^= 1u;
            at.slot = at.slot == 0 ? a.n_stages - 1 : at.slot - 1;
            mbar_wait(full + 8 * at.slot, at.phase, nullptr, TC_WAIT_LIMIT >> 6);
        }
    }
};

// ------------------------------------------------------------------------------------------------- consumers
struct Consumer {
    const StackArgs& a;
    Shared& sh;
    float* scratch;        // partial sums of the warps; of attention: their outputs
    unsigned char* ring_mem;
    uint32_t full, empty;
    int tid, lane, warp, g, t;
    Ring at;

    // Hides from the compiler that these are the same in every phase: it would keep what all phases work out from them in registers throughout.
    __device__ __forceinline__ void forget() { asm volatile("" : "+r"(tid), "+r"(lane), "+r"(warp), "+r"(g), "+r"(t)); }
    __device__ __forceinline__ void wait_stage() { wait_bar(full + 8 * at.slot, at.phase, sh, a.status); }
    __device__ __forceinline__ void release() {
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * at.slot);
        at.next(a.n_stages);
    }
    // A lane's 16 elements of row g of a stage, 32 bytes: x of a half of the warp's part of the contraction in the same order.  Odd rows
    // are read with their two halves the other way round: the eight lanes of a pass then meet all banks once.
    __device__ __forceinline__ void fragment(uint4& u0, uint4& u1, const unsigned char* p) const {
        const bool odd = g & 1;
        const uint4 a0 = reinterpret_cast<const uint4*>(p)[odd], a1 = reinterpret_cast<const uint4*>(p)[!odd];
        u0 = odd ? a1 : a0, u1 = odd ? a0 : a1;
    }
    // A tile's two stages (or its only one): the warp's part of the contraction for sixteen rows.  x: elements 16 t ... 16 t + 15 of
    // token g's 64 and the next 64, two a register.  Not `live`: the contraction ends before this warp's part, where the stage holds
    // what it held before.
    __device__ __forceinline__ void tile_mma(float (&c0)[4], float (&c1)[4], const uint32_t (&x)[16], bool second, int live) {
        const unsigned char* mine = ring_mem + g * ROW_BYTES + warp * (KW * 2) + t * 32;
        const int slot0 = at.slot;
        wait_stage();
        at.next(a.n_stages);
        const int slot1 = at.slot;
        if (second) wait_stage();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i >= live) break;
            uint4 u0, u1, v0 = make_uint4(0u, 0u, 0u, 0u), v1 = v0;
            fragment(u0, u1, mine + slot0 * STAGE_BYTES + 128 * i);
            if (second) fragment(v0, v1, mine + slot1 * STAGE_BYTES + 128 * i);
            mma(c0, u0.x, v0.x, u0.y, v0.y, x[8 * i], x[8 * i + 1]);
            mma(c1, u0.z, v0.z, u0.w, v0.w, x[8 * i + 2], x[8 * i + 3]);
            mma(c0, u1.x, v1.x, u1.y, v1.y, x[8 * i + 4], x[8 * i + 5]);
            mma(c1, u1.z, v1.z, u1.w, v1.w, x[8 * i + 6], x[8 * i + 7]);
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(empty + 8 * slot0);
            if (second) mbar_arrive(empty + 8 * slot1);
        }
        if (second) at.next(a.n_stages);
    }
    __device__ __forceinline__ int live(int chunk, int K) const { return (K - chunk * KC - warp * KW) / 64; }   // 64s of the warp's part there are
    // Sums of a tile: [row][token].
    __device__ __forceinline__ void put_sums(int slot, const float (&c0)[4], const float (&c1)[4]) {
        if (2 * t < a.T) {
            float* p = scratch + (slot * CW + warp) * (TILE * MAX_T) + g * MAX_T + 2 * t;
            *reinterpret_cast<float2*>(p) = make_float2(c0[0] + c1[0], c0[1] + c1[1]);
            *reinterpret_cast<float2*>(p + ROWS * MAX_T) = make_float2(c0[2] + c1[2], c0[3] + c1[3]);
        }
    }
    __device__ __forceinline__ float warp_sums(int slot, int e) const {
        const float* p = scratch + slot * CW * (TILE * MAX_T) + e;
        float v[CW], s = 0.f;
#pragma unroll
        for (int w = 0; w < CW; ++w) v[w] = p[w * (TILE * MAX_T)];
#pragma unroll
        for (int w = 0; w < CW; ++w) s += v[w];
        return s;
    }
    // bfloat16 x [T, K]: the warp's elements of part `chunk`.
    __device__ __forceinline__ void load_x(uint32_t (&x)[16], const __nv_bfloat16* src, int K, int chunk) const {
        const int k = chunk * KC + warp * KW;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint4 u = make_uint4(0u, 0u, 0u, 0u), v = u;
            if (g < a.T && k + 64 * i < K) {
                const uint4* p = reinterpret_cast<const uint4*>(src + g * K + k + 64 * i + 16 * t);
                u = __ldcg(p), v = __ldcg(p + 1);
            }
            x[8 * i] = u.x, x[8 * i + 1] = u.y, x[8 * i + 2] = u.z, x[8 * i + 3] = u.w, x[8 * i + 4] = v.x, x[8 * i + 5] = v.y, x[8 * i + 6] = v.z, x[8 * i + 7] = v.w;
        }
    }
    // x = rmsnorm(h) * w, from the shares of the sums of squares.  The stream is asked for before the sums are there.
    template <int XS>
    __device__ __forceinline__ void norm_x(uint32_t (&x)[XS][16], const float* w, float eps) {
        float s = 0.f;
        if (warp < a.T)
            for (int i = lane; i < (int)gridDim.x; i += 32) s += __ldcg(a.ss + warp * STACK_SS_STRIDE + i);
#pragma unroll
        for (int c = 0; c < XS; ++c) {
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = c * KC + warp * KW + 64 * (j / 4);
                v[j] = g < a.T && k < a.d ? __ldcg(reinterpret_cast<const float4*>(a.h + g * a.d + k + 16 * t) + j % 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            if (c == 0) {
                s = warp_sum(s);
                if (lane == 0 && warp < a.T) sh.inv[warp] = rsqrtf(s / (float)a.d + eps);
                consumers_sync();
            }
            const float inv = g < a.T ? sh.inv[g] : 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int k = c * KC + warp * KW + 64 * (j / 4);
                float4 wv = make_float4(0.f, 0.f, 0.f, 0.f);
                if (g < a.T && k < a.d) wv = __ldg(reinterpret_cast<const float4*>(w + k + 16 * t) + j % 4);
                x[c][2 * j] = pack(v[j].x * inv * wv.x, v[j].y * inv * wv.y);
                x[c][2 * j + 1] = pack(v[j].z * inv * wv.z, v[j].w * inv * wv.w);
            }
        }
    }

    // Phases 1 and 4.
    template <int XS>
    __device__ __forceinline__ void normed_product(const float* norm_w, float eps, int r0, int r1, bool gated, __nv_bfloat16* out, int ld) {
        forget();
        uint32_t x[XS][16];
        norm_x(x, norm_w, eps);
        const int per = gated ? ROWS : TILE, n_tiles = (r1 - r0 + per - 1) / per, chunks = (a.d + KC - 1) / KC;
        const int slot = tid / (TILE * MAX_T), e = tid % (TILE * MAX_T), tok = e % MAX_T, j = e / MAX_T;
        for (int b = 0; b < n_tiles; b += BATCH) {
            const int n = min(BATCH, n_tiles - b);
            for (int i = 0; i < n; ++i) {
                float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
                const bool second = gated || r0 + (b + i) * TILE + ROWS < r1;
#pragma unroll
                for (int c = 0; c < XS; ++c)
                    if (c < chunks) tile_mma(c0, c1, x[c], second, live(c, a.d));
                put_sums(i, c0, c1);
            }
            consumers_sync();
            for (int i = slot; i < n; i += SLOTS) {
                const int r = r0 + (b + i) * per + j;
                if (j < per && r < r1 && tok < a.T) {
                    float v = warp_sums(i, e);
                    if (gated) v = gated_f(v, warp_sums(i, e + ROWS * MAX_T), GateAct(a.act, a.act_limit));
                    out[tok * ld + r] = __float2bfloat16_rn(v);
                }
            }
            if (b + BATCH < n_tiles) consumers_sync();   // the sums have been read
        }
    }

    // Phases 3 and 5: h += x W^T for the columns r0 ... r1 - 1 of the stream; their squares' sum goes to a.ss.
    __device__ __forceinline__ void branch_product(const __nv_bfloat16* src, int K, int r0, int r1) {
        forget();
        const int n_tiles = (r1 - r0 + TILE - 1) / TILE, chunks = (K + KC - 1) / KC;
        uint32_t x[BX][16];
#pragma unroll
        for (int c = 0; c < BX; ++c) load_x(x[c], src, K, c);
        const int slot = tid / (TILE * MAX_T), e = tid % (TILE * MAX_T), tok = e % MAX_T, r = r0 + slot * TILE + e / MAX_T;
        constexpr int OUT = (TILES + SLOTS - 1) / SLOTS;   // outputs of a thread
        float old[OUT];
#pragma unroll
        for (int i = 0; i < OUT; ++i) old[i] = tok < a.T && r + i * SLOTS * TILE < r1 ? __ldcg(a.h + tok * a.d + r + i * SLOTS * TILE) : 0.f;
        float c[TILES][4];
#pragma unroll
        for (int i = 0; i < TILES; ++i) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
#pragma unroll 1
        for (int base = 0; base < chunks; base += BX) {
#pragma unroll
            for (int k = 0; k < BX; ++k) {
                if (base + k >= chunks) break;
#pragma unroll
                for (int i = 0; i < TILES; ++i)
                    if (i < n_tiles) tile_mma(c[i], c[i], x[k], r0 + i * TILE + ROWS < r1, live(base + k, K));
                if (base + k + BX < chunks) load_x(x[k], src, K, base + k + BX);
            }
        }
        const float none[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < TILES; ++i)
            if (i < n_tiles) put_sums(i, c[i], none);
        consumers_sync();
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < OUT; ++i)
            if (tok < a.T && r + i * SLOTS * TILE < r1) {
                const float v = old[i] + __bfloat162float(__float2bfloat16_rn(warp_sums(slot + i * SLOTS, e)));
                __stcg(a.h + tok * a.d + r + i * SLOTS * TILE, v);
                sq += v * v;
            }
        put_squares(sq);
    }
    // The CTA's share of every row's sum of squares, from its threads' (token tid % MAX_T).
    __device__ __forceinline__ void put_squares(float sq) {
        sq += __shfl_xor_sync(0xffffffffu, sq, 8);
        sq += __shfl_xor_sync(0xffffffffu, sq, 16);
        if (lane < MAX_T) sh.ss[warp][lane] = sq;
        consumers_sync();
        if (tid < a.T) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < CW; ++w) s += sh.ss[w][tid];
            __stcg(a.ss + tid * STACK_SS_STRIDE + blockIdx.x, s);
        }
    }
    // The sums of squares of the stream as it comes in.
    __device__ __forceinline__ void first_squares(int r0, int r1) {
        const int tok = tid % MAX_T;
        float sq = 0.f;
        for (int r = r0 + tid / MAX_T; r < r1 && tok < a.T; r += CT / MAX_T) {
            const float v = __ldcg(a.h + tok * a.d + r);
            sq += v * v;
        }
        put_squares(sq);
    }

    // Phase 2.
    __device__ __forceinline__ void attention(const StackLayer& L) {
        forget();
        const int G = a.hq / a.hkv, n_items = sh.item0[a.T], qkv_ld = (a.hq + 2 * a.hkv) * DH;
        for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
            const Item it = item_of(sh, item, a.T);
            const int pos = sh.pos[it.tok], n_units = it.unit1 - it.unit0, n_warps = min(CW, n_units);
            const __nv_bfloat16* row = a.qkv + (int64_t)it.tok * qkv_ld;
            const float* cs = a.cos_tab + (int64_t)pos * (DH / 2);
            const float* sn = a.sin_tab + (int64_t)pos * (DH / 2);
            uint32_t q[4][4];         // block b: dimensions 32 b + 8 t ... + 7 of head g
            float o[8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};   // heads 2 t and 2 t + 1
            const bool own = it.part == it.parts - 1 && (n_units - 1) % CW == warp;   // the last block holds the token's own key
            if (warp < n_warps) {
                load_q(q, row + (int64_t)(it.kvh * G + g) * DH, g < G, L.q_norm, cs, sn);
                if (own) make_own(row, it, pos, L, cs, sn);
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
            }
            for (int u = 0; u < n_units; ++u) {
                wait_stage();
                if (u % CW != warp) {    // passed by all the same: a stage is refilled when every warp has seen it
                    release();
                    continue;
                }
                unsigned char* ksm = ring_mem + at.slot * STAGE_BYTES;
                unsigned char* vsm = ksm + 2 * RUN_BYTES;
                const int j0 = (it.unit0 + u) * UNIT;
                if (own && u == n_units - 1) {
                    const int r = pos - j0;
                    reinterpret_cast<uint2*>(ksm + r * DH * 2)[lane] = reinterpret_cast<const uint2*>(sh.own_k)[lane];
                    reinterpret_cast<uint2*>(vsm + r * DH * 2)[lane] = reinterpret_cast<const uint2*>(sh.own_v)[lane];
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // a copy refills the stage later
                    __syncwarp();
                }
                keys32(q, o, m, l, ksm, vsm, j0, pos);
                release();
            }
            if (warp < n_warps) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int x = 4; x < 32; x <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], x);
                    if (2 * t + h >= G) continue;
                    float* dst = scratch + (warp * G + 2 * t + h) * DH + 8 * g;     // [warp][head][DH]
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        *reinterpret_cast<float4*>(dst + 64 * b) = make_float4(o[4 * b][h], o[4 * b][2 + h], o[4 * b + 1][h], o[4 * b + 1][2 + h]);
                        *reinterpret_cast<float4*>(dst + 64 * b + 4) = make_float4(o[4 * b + 2][h], o[4 * b + 2][2 + h], o[4 * b + 3][h], o[4 * b + 3][2 + h]);
                    }
                    if (g == 0) sh.m[warp][2 * t + h] = m[h], sh.l[warp][2 * t + h] = l[h];
                }
            }
            consumers_sync();
            merge(item, n_warps);
            if (item + (int)gridDim.x < n_items) consumers_sync();   // the scratch has been read
        }
    }
    // The warps' outputs of an item into one, and, in the CTA that comes last, those of the item's (token, kv head).
    __device__ __forceinline__ void merge(int item, int n_warps) {
        const int G = a.hq / a.hkv;
        const Item it = item_of(sh, item, a.T);
        __nv_bfloat16* out = a.attn + (int64_t)it.tok * a.hq * DH + (int64_t)it.kvh * G * DH;
        for (int e = tid; e < G * DH; e += CT) {
            const int h = e / DH;
            float M = -INFINITY, s = 0.f, L = 0.f;
            for (int w = 0; w < n_warps; ++w) M = fmaxf(M, sh.m[w][h]);
            for (int w = 0; w < n_warps; ++w) {
                const float f = exp2f(sh.m[w][h] - M);
                s += scratch[w * G * DH + e] * f;
                L += sh.l[w][h] * f;
            }
            if (it.parts == 1) {
                out[e] = __float2bfloat16_rn(s * (1.f / L));
            } else {
                __stcg(a.part_o + (int64_t)item * G * DH + e, s);
                if (e % DH == 0) __stcg(reinterpret_cast<float2*>(a.part_ml) + (int64_t)item * G + h, make_float2(M, L));
            }
        }
        if (it.parts == 1) return;
        consumers_sync();
        if (tid == 0) {
            unsigned* count = a.sync + 2 + it.tok * a.hkv + it.kvh;
            __threadfence();
            const bool last = atomicAdd(count, 1u) == (unsigned)it.parts - 1;
            sh.last = last;
            if (last) *reinterpret_cast<volatile unsigned*>(count) = 0u;
            __threadfence();
        }
        consumers_sync();
        if (!sh.last) return;
        const int first = item - it.part;
        for (int e = tid; e < G * DH; e += CT) {
            const int h = e / DH;
            float M = -INFINITY, s = 0.f, L = 0.f;
            for (int p0 = 0; p0 < it.parts; p0 += 8) {     // eight parts on their way at a time, added in part order
                float2 ml[8];
                float v[8];
#pragma unroll
                for (int p = 0; p < 8; ++p)
                    if (p0 + p < it.parts) {
                        ml[p] = __ldcg(reinterpret_cast<const float2*>(a.part_ml) + (int64_t)(first + p0 + p) * G + h);
                        v[p] = __ldcg(a.part_o + (int64_t)(first + p0 + p) * G * DH + e);
                    }
                float top = M;
#pragma unroll
                for (int p = 0; p < 8; ++p)
                    if (p0 + p < it.parts) top = fmaxf(top, ml[p].x);
                const float f0 = exp2f(M - top);
                s *= f0;
                L *= f0;
                M = top;
#pragma unroll
                for (int p = 0; p < 8; ++p)
                    if (p0 + p < it.parts) {
                        const float f = exp2f(ml[p].x - M);
                        s += v[p] * f;
                        L += ml[p].y * f;
                    }
            }
            out[e] = __float2bfloat16_rn(s * (1.f / L));
        }
    }
    // Head g's query as the right operand: normalised, rotated (pairs d, d + 64: blocks b and b + 2 of the same lane).
    __device__ __forceinline__ void load_q(uint32_t (&qa)[4][4], const __nv_bfloat16* q, bool used, const float* norm_w, const float* cs, const float* sn) const {
        float2 v[4][4];
        float ss = 0.f;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint4 u = used ? __ldcg(reinterpret_cast<const uint4*>(q + 32 * b + 8 * t)) : make_uint4(0u, 0u, 0u, 0u);
            v[b][0] = unpack(u.x), v[b][1] = unpack(u.y), v[b][2] = unpack(u.z), v[b][3] = unpack(u.w);
#pragma unroll
            for (int j = 0; j < 4; ++j) ss += v[b][j].x * v[b][j].x + v[b][j].y * v[b][j].y;
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (norm_w) {
            const float inv = rsqrtf(ss / (float)DH + a.qk_eps);
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 w = __ldg(reinterpret_cast<const float2*>(norm_w + 32 * b + 8 * t + 2 * j));
                    v[b][j].x = v[b][j].x * inv * w.x;
                    v[b][j].y = v[b][j].y * inv * w.y;
                }
        }
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 c = __ldg(reinterpret_cast<const float2*>(cs + 32 * b + 8 * t + 2 * j)), s = __ldg(reinterpret_cast<const float2*>(sn + 32 * b + 8 * t + 2 * j));
                const float2 x = v[b][j], y = v[b + 2][j];
                qa[b][j] = pack(x.x * c.x - y.x * s.x, x.y * c.y - y.y * s.y);
                qa[b + 2][j] = pack(x.x * s.x + y.x * c.x, x.y * s.y + y.y * c.y);
            }
    }
    // The token's own key and value, written to their page and kept for the copy in shared memory.
    __device__ __forceinline__ void make_own(const __nv_bfloat16* row, const Item& it, int pos, const StackLayer& L, const float* cs, const float* sn) const {
        const __nv_bfloat16* k = row + (int64_t)(a.hq + it.kvh) * DH;
        const __nv_bfloat16* v = k + (int64_t)a.hkv * DH;
        float2 x = unpack(__ldcg(reinterpret_cast<const uint32_t*>(k) + lane)), y = unpack(__ldcg(reinterpret_cast<const uint32_t*>(k + DH / 2) + lane));
        const uint2 val = __ldcg(reinterpret_cast<const uint2*>(v) + lane);
        const float ss = warp_sum(x.x * x.x + x.y * x.y + y.x * y.x + y.y * y.y);
        if (L.k_norm) {
            const float inv = rsqrtf(ss / (float)DH + a.qk_eps);
            const float2 w0 = __ldg(reinterpret_cast<const float2*>(L.k_norm) + lane), w1 = __ldg(reinterpret_cast<const float2*>(L.k_norm + DH / 2) + lane);
            x.x = x.x * inv * w0.x, x.y = x.y * inv * w0.y;
            y.x = y.x * inv * w1.x, y.y = y.y * inv * w1.y;
        }
        const float2 c = __ldg(reinterpret_cast<const float2*>(cs) + lane), s = __ldg(reinterpret_cast<const float2*>(sn) + lane);
        const uint32_t lo = pack(x.x * c.x - y.x * s.x, x.y * c.y - y.y * s.y), hi = pack(x.x * s.x + y.x * c.x, x.y * s.y + y.y * c.y);
        sh.own_k[lane] = lo;
        sh.own_k[32 + lane] = hi;
        reinterpret_cast<uint2*>(sh.own_v)[lane] = val;
        __syncwarp();
        const int page = a.block_table[(int64_t)sh.seq[it.tok] * a.bt_stride + pos / a.page_size];
        if (page < 0 || page >= a.num_pages) return;   // the producer reports it
        const int64_t off = (((int64_t)page * a.hkv + it.kvh) * a.page_size + pos % a.page_size) * DH;
        reinterpret_cast<uint32_t*>((__nv_bfloat16*)L.k_pages + off)[lane] = lo;
        reinterpret_cast<uint32_t*>((__nv_bfloat16*)L.k_pages + off + DH / 2)[lane] = hi;
        reinterpret_cast<uint2*>((__nv_bfloat16*)L.v_pages + off)[lane] = val;
    }
    // Scores, softmax update and P V for 32 keys from position j0 on (16 where the others lie behind the token).  Keys and dimensions
    // are the tensor operation's 16 rows, query heads its 8 columns.
    __device__ __forceinline__ void keys32(const uint32_t (&q)[4][4], float (&o)[8][4], float (&m)[2], float (&l)[2], const unsigned char* ksm,
                                           const unsigned char* vsm, int j0, int pos) const {
        const bool odd = g & 1, both = j0 + 16 <= pos;
        float s[2][4];      // keys j0 + 16 i + g and + 8, heads 2 t and 2 t + 1
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
            if (i == 1 && !both) continue;
            const unsigned char* p = ksm + i * RUN_BYTES + g * (DH * 2) + t * 16;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                // odd keys ask for the blocks of 64 bytes in the other order: the eight lanes of a pass then meet all banks once
                const unsigned char* p0 = p + half * 128 + (odd ? 64 : 0);
                const unsigned char* p1 = p + half * 128 + (odd ? 0 : 64);
                const uint4 a0 = *reinterpret_cast<const uint4*>(p0), a1 = *reinterpret_cast<const uint4*>(p1);
                const uint4 b0 = *reinterpret_cast<const uint4*>(p0 + 8 * DH * 2), b1 = *reinterpret_cast<const uint4*>(p1 + 8 * DH * 2);
                const uint4 x0 = odd ? a1 : a0, x1 = odd ? a0 : a1, y0 = odd ? b1 : b0, y1 = odd ? b0 : b1;
                mma(s[i], x0.x, y0.x, x0.y, y0.y, q[2 * half][0], q[2 * half][1]);
                mma(s[i], x0.z, y0.z, x0.w, y0.w, q[2 * half][2], q[2 * half][3]);
                mma(s[i], x1.x, y1.x, x1.y, y1.y, q[2 * half + 1][0], q[2 * half + 1][1]);
                mma(s[i], x1.z, y1.z, x1.w, y1.w, q[2 * half + 1][2], q[2 * half + 1][3]);
            }
        }
        float corr[2], top[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float& v = s[i][2 * r + h];
                    v = j0 + 16 * i + 8 * r + g <= pos ? v * a.scale_log2 : -INFINITY;
                    mx = fmaxf(mx, v);
                }
#pragma unroll
            for (int x = 4; x < 32; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            const float m_new = fmaxf(m[h], mx);
            top[h] = m_new == -INFINITY ? 0.f : m_new;
            corr[h] = exp2_fast(m[h] - top[h]);
            m[h] = m_new;
            l[h] *= corr[h];
        }
        uint32_t p[2][2];   // run of 16 keys, eight of them: head g, keys 2 t and 2 t + 1
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float e0 = exp2_fast(s[i][2 * r] - top[0]), e1 = exp2_fast(s[i][2 * r + 1] - top[1]);
                l[0] += e0;
                l[1] += e1;
                p[i][r] = transposed(pack(e0, e1));
            }
        if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i][0] *= corr[0], o[i][1] *= corr[1], o[i][2] *= corr[0], o[i][3] *= corr[1];
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i == 1 && !both) continue;
            const unsigned char* vr = vsm + i * RUN_BYTES + 2 * t * (DH * 2) + 16 * g;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint4 r0 = *reinterpret_cast<const uint4*>(vr + b * 128), r1 = *reinterpret_cast<const uint4*>(vr + DH * 2 + b * 128);
                const uint4 r2 = *reinterpret_cast<const uint4*>(vr + 16 * DH + b * 128), r3 = *reinterpret_cast<const uint4*>(vr + 18 * DH + b * 128);
                const uint32_t w0[4] = {r0.x, r0.y, r0.z, r0.w}, w1[4] = {r1.x, r1.y, r1.z, r1.w}, w2[4] = {r2.x, r2.y, r2.z, r2.w}, w3[4] = {r3.x, r3.y, r3.z, r3.w};
#pragma unroll
                for (int k = 0; k < 4; ++k)   // rows g: dimension 64 b + 8 g + 2 k, rows g + 8: the next one
                    mma(o[4 * b + k], __byte_perm(w0[k], w1[k], 0x5410u), __byte_perm(w0[k], w1[k], 0x7632u), __byte_perm(w2[k], w3[k], 0x5410u),
                        __byte_perm(w2[k], w3[k], 0x7632u), p[i][0], p[i][1]);
            }
        }
    }
};

// Everybody's stores before, everybody's loads after.  All consumer threads call it; `target`: arrivals of all CTAs so far and at this one.
__device__ __forceinline__ void grid_sync(const StackArgs& a, Shared& sh, unsigned target) {
    consumers_sync();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.sync) : "memory");
        for (uint32_t i = 0;; ++i) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.sync) : "memory");
            if (v >= target || sh.dead) break;
            if (i == TC_WAIT_LIMIT) {
                sh.dead = 1;
                imp_report(a.status, IMP_WAIT_TIMEOUT);
                break;
            }
        }
        __threadfence();
    }
    consumers_sync();
}

// A line of a small vector that everybody reads two phases from now: asked into the L2 by one CTA.
__device__ __forceinline__ void ask(const float* p, int n, int tid) {
    if (p && tid == 0 && (int)blockIdx.x * 32 < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + blockIdx.x * 32));
    if (p && tid == 32 && (int)(blockIdx.x + gridDim.x) * 32 < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + (blockIdx.x + gridDim.x) * 32));
}

template <int XS>
__global__ void __launch_bounds__(THREADS, 1) decode_stack_kernel(const __grid_constant__ StackArgs a) {
    Shared& sh = *reinterpret_cast<Shared*>(stack_smem);
    StackLayer* layers = reinterpret_cast<StackLayer*>(stack_smem + SHARED_BYTES);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t full = smem_u32(sh.full), empty = smem_u32(sh.empty);
    for (int i = tid; i < a.n_layers * (int)(sizeof(StackLayer) / 8); i += THREADS)
        reinterpret_cast<uint64_t*>(layers)[i] = reinterpret_cast<const uint64_t*>(a.layers)[i];
    if (tid < a.T) {
        sh.pos[tid] = a.positions[tid];
        sh.seq[tid] = a.seq_of_token[tid];
    }
    if (tid == 0) {
        sh.dead = 0;
        for (int i = 0; i < a.n_stages; ++i) {
            mbar_init(full + 8 * i, 1);
            mbar_init(empty + 8 * i, CW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    bool good = true;      // the same for everybody
    for (int t = 0; t < a.T; ++t) {
        const int p = sh.pos[t], s = sh.seq[t];
        if (s < 0 || s >= a.n_seqs) {
            good = false;
            if (tid == 0) imp_report(a.status, IMP_BAD_SEQUENCE);
        } else if (p < 0 || p / a.page_size >= a.bt_stride || p >= a.max_pos) {
            good = false;
            if (tid == 0) imp_report(a.status, IMP_BAD_POSITION);
        }
    }
    if (!good) return;
    if (tid == 0) {
        // Parts of the keys: the fewest blocks a part (at least MIN_UNITS) with which the items do not outnumber the CTAs.
        int total = 0, longest = 0;
        for (int t = 0; t < a.T; ++t) {
            sh.units[t] = sh.pos[t] / UNIT + 1;
            total += sh.units[t];
            longest = max(longest, sh.units[t]);
        }
        int most = max(MIN_UNITS, (int)(((int64_t)total * a.hkv + gridDim.x - 1) / gridDim.x));
        for (; most < longest; ++most) {
            int items = 0;
            for (int t = 0; t < a.T; ++t) items += (sh.units[t] + most - 1) / most;
            if (items * a.hkv <= (int)gridDim.x) break;
        }
        int items = 0;
        for (int t = 0; t < a.T; ++t) {
            sh.item0[t] = items;
            sh.parts[t] = (sh.units[t] + most - 1) / most;
            items += sh.parts[t] * a.hkv;
        }
        sh.item0[a.T] = items;
    }
    __syncthreads();
    const int cta = blockIdx.x, ctas = gridDim.x, qkv = (a.hq + 2 * a.hkv) * DH;
    const int qkv0 = share(qkv, cta, ctas), qkv1 = share(qkv, cta + 1, ctas);
    const int d0 = share(a.d, cta, ctas), d1 = share(a.d, cta + 1, ctas), f0 = share(a.F, cta, ctas), f1 = share(a.F, cta + 1, ctas);
    // 384 threads are launched with 168 registers each, 64,512; of these 256 take 224 and 128 keep 56.
    if (warp >= CW) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == CW) {
            Producer p{a, sh, smem_u32(stack_smem + a.ring_at), full, empty, lane};
            for (int i = 0; i < a.n_layers && p.ok; ++i) {
                const StackLayer& L = layers[i];
                p.by_tile((const __nv_bfloat16*)L.w_qkv, qkv0, qkv1, a.d, false);
                p.keys(L);
                p.by_chunk((const __nv_bfloat16*)L.w_o, d0, d1, a.hq * DH);
                p.by_tile((const __nv_bfloat16*)L.w_gu, f0, f1, a.d, true);
                p.by_chunk((const __nv_bfloat16*)L.w_down, d0, d1, a.F);
            }
            p.drain();
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        Consumer c{a, sh, reinterpret_cast<float*>(stack_smem + a.scratch_at), stack_smem + a.ring_at, full, empty, tid, lane, warp, lane >> 2, lane & 3};
        unsigned arrived = ctas;
        c.first_squares(d0, d1);
        grid_sync(a, sh, arrived);
        for (int i = 0; i < a.n_layers; ++i) {
            const StackLayer& L = layers[i];
            c.normed_product<XS>(L.norm1, a.eps1, qkv0, qkv1, false, a.qkv, qkv);
            ask(L.norm2, a.d, tid);
            grid_sync(a, sh, arrived += ctas);
            c.attention(L);
            grid_sync(a, sh, arrived += ctas);
            c.branch_product(a.attn, a.hq * DH, d0, d1);
            grid_sync(a, sh, arrived += ctas);
            c.normed_product<XS>(L.norm2, a.eps2, f0, f1, true, a.hid, a.F);
            if (i + 1 < a.n_layers) {
                ask(layers[i + 1].norm1, a.d, tid);
                ask(layers[i + 1].q_norm, DH, tid);
                ask(layers[i + 1].k_norm, DH, tid);
            }
            grid_sync(a, sh, arrived += ctas);
            c.branch_product(a.hid, a.F, d0, d1);
            if (i + 1 < a.n_layers) grid_sync(a, sh, arrived += ctas);
        }
    }
    __syncthreads();
    // The last CTA leaves the counters as it found them, whatever happened.
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(a.sync + 1, 1u) == gridDim.x - 1) {
            for (int i = 0; i < 2 + a.T * a.hkv; ++i) a.sync[i] = 0u;
            __threadfence();
        }
    }
}

constexpr int MOST_SMEM = 232448;
template <int XS>
int launch(const StackArgs& a, int ctas, size_t smem, cudaStream_t stream) {
    static bool ready[64] = {};   // the attribute is a property of the function on a device; setting it twice does no harm
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return IMP_ERR_UNSUPPORTED;
    if (!ready[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(decode_stack_kernel<XS>, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM);
        if (e != cudaSuccess) {
            imp_set_error("decode_stack: %s", cudaGetErrorString(e));
            return (int)e;
        }
        ready[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;    // all CTAs at once or none: they wait for one another
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_stack_kernel<XS>, a);
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // part of the device only
        (void)cudaGetLastError();
        return IMP_ERR_UNSUPPORTED;
    }
    if (e != cudaSuccess) {
        imp_set_error("decode_stack: %s", cudaGetErrorString(e));
        return (int)e;
    }
    return 0;
}

int stack_ctas() { return imp_sm_count(); }
}  // namespace

IMP_API int imp_decode_stack_items(int T, int hkv) { return T * hkv > stack_ctas() ? T * hkv : stack_ctas(); }

IMP_API int imp_decode_stack_supported(int d, int F, int hq, int hkv, int dh, int page_size, int n_layers) {
    const int ctas = stack_ctas();
    if (ctas < 1 || ctas > STACK_SS_STRIDE || dh != DH || hkv <= 0 || hq % hkv || hq / hkv > 8) return 0;
    if (d <= 0 || d % 64 || d > 6 * KC || F <= 0 || F % 64 || page_size <= 0 || page_size % 16 || n_layers <= 0 || n_layers > STACK_MAX_LAYERS) return 0;
    return (d + ctas - 1) / ctas <= TILES * TILE;
}

IMP_API int imp_decode_stack(const StackArgs* args, void* stream) {
    StackArgs a = *args;
    IMP_CHECK_ARG(a.layers && a.h && a.qkv && a.attn && a.hid && a.ss && a.part_o && a.part_ml && a.sync && a.positions && a.seq_of_token && a.block_table &&
                      a.cos_tab && a.sin_tab,
                  "decode_stack: null argument");
    IMP_CHECK_ARG(a.T > 0 && a.n_seqs > 0, "decode_stack: no tokens");
    if (a.T > MAX_T || !imp_decode_stack_supported(a.d, a.F, a.hq, a.hkv, DH, a.page_size, a.n_layers)) return IMP_ERR_UNSUPPORTED;
    const int G = a.hq / a.hkv;
    const int sums = BATCH * CW * TILE * MAX_T * 4, outputs = CW * G * DH * 4;
    a.scratch_at = (SHARED_BYTES + a.n_layers * (int)sizeof(StackLayer) + 127) / 128 * 128;
    a.ring_at = a.scratch_at + (sums > outputs ? sums : outputs);
    const int fit = (MOST_SMEM - a.ring_at) / STAGE_BYTES;
    a.n_stages = fit < MAX_STAGES ? fit : MAX_STAGES;
    if (a.n_stages < 4) return IMP_ERR_UNSUPPORTED;
    const size_t smem = (size_t)a.ring_at + (size_t)a.n_stages * STAGE_BYTES;
    const int xs = (a.d + KC - 1) / KC, ctas = stack_ctas();
    cudaStream_t s = (cudaStream_t)stream;
    if (xs <= 1) return launch<1>(a, ctas, smem, s);
    if (xs <= 2) return launch<2>(a, ctas, smem, s);
    if (xs <= 4) return launch<4>(a, ctas, smem, s);
    return launch<6>(a, ctas, smem, s);
}
