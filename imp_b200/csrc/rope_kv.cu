// Per-head RMSNorm on q and k, rotary position encoding, and the write of k and
// v into the paged cache, in one pass over the fused q|k|v projection output.
//
// Reference counterparts: rmsnorm on q/k viewed per head (src/graph/
// executor_forward.cu:537-546), rope_forward_* (src/compute/rope.cu:45-182),
// the fused decode kernel (src/compute/rope.cu:270-413) and
// write_kv_cache_fused_kernel (src/graph/executor_kernels.cu:342-388).
// Pairing is (i, i + rot/2) ("neox"), x_i' = x_i cos a - x_{i+rot/2} sin a,
// x_{i+rot/2}' = x_i sin a + x_{i+rot/2} cos a (src/compute/rope.cu:96-101).
// Differences: cos and sin come from a table built in double precision on the
// host (the reference evaluates __cosf/__sinf of a 32-bit angle), the norm's
// result stays in 32-bit until after the rotation, and any number of tokens of
// any mix of sequences is handled by one launch (the reference's cache write
// assumes token i belongs to sequence i in a batch).
//
// Cache layout of one layer: K and V each [num_pages][kv_heads][page_size][head_dim].
#include "common.cuh"

template <typename TA, typename TW>
__global__ void qk_norm_rope_kv_kernel(
    TA* __restrict__ qkv, int64_t row_stride, int Hq, int Hkv, int Dh,
    const TW* __restrict__ q_norm_w, const TW* __restrict__ k_norm_w, float eps, float weight_offset,
    const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int rot_dim, int max_pos,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ block_table, int bt_stride, int n_seqs,
    TA* __restrict__ k_cache, TA* __restrict__ v_cache, int page_size, int num_pages,
    int n_tokens, int* status) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int heads_per_token = Hq + 2 * Hkv;
    if (unit >= n_tokens * heads_per_token) return;
    const int t = unit / heads_per_token;
    const int hh = unit - t * heads_per_token;
    const int pos = positions[t];
    TA* x = qkv + (int64_t)t * row_stride + (int64_t)hh * Dh;

    const bool is_q = hh < Hq;
    const bool is_k = !is_q && hh < Hq + Hkv;
    const int kv_head = is_q ? 0 : (is_k ? hh - Hq : hh - Hq - Hkv);

    // Where this head's row lives in the cache (k and v only).
    TA* dst = nullptr;
    if (!is_q) {
        TA* cache = is_k ? k_cache : v_cache;
        if (cache == nullptr) {
            if (!is_k) return;  // v without a cache: nothing to do
        } else {
            const int seq = seq_of_token[t];
            if (seq < 0 || seq >= n_seqs) {
                if (lane == 0) imp_report(status, IMP_BAD_SEQUENCE);
                return;
            }
            const int slot_page = pos / page_size;
            if (pos < 0 || slot_page >= bt_stride) {
                if (lane == 0) imp_report(status, IMP_TAGGED(IMP_BAD_POSITION, 6));
                return;
            }
            const int page = block_table[(int64_t)seq * bt_stride + slot_page];
            if (page < 0 || page >= num_pages) {
                if (lane == 0) imp_report(status, IMP_BAD_PAGE);
                return;
            }
            dst = cache + (((int64_t)page * Hkv + kv_head) * page_size + (pos - slot_page * page_size)) * Dh;
        }
    }

    if (!is_q && !is_k) {  // v: plain copy into its page
        for (int i = lane; i < Dh; i += 32) dst[i] = x[i];
        return;
    }

    const TW* nw = is_q ? q_norm_w : k_norm_w;
    float inv = 1.f;
    if (nw) {
        float ss = 0.f;
        for (int i = lane; i < Dh; i += 32) {
            const float v = to_float(x[i]);
            ss += v * v;
        }
        ss = warp_sum(ss);
        inv = rsqrtf(ss / (float)Dh + eps);
    }
    const int half = rot_dim >> 1;
    const bool rotate = cos_tab != nullptr && half > 0;
    if (rotate && (pos < 0 || pos >= max_pos)) {
        if (lane == 0) imp_report(status, IMP_TAGGED(IMP_BAD_POSITION, 6));
        return;
    }
    TA* out = is_q ? x : (dst ? dst : x);
    // Rotated part: pairs (i, i + half).
    for (int i = lane; i < half; i += 32) {
        float a = to_float(x[i]) * inv, b = to_float(x[i + half]) * inv;
        if (nw) {
            a *= to_float(nw[i]) + weight_offset;
            b *= to_float(nw[i + half]) + weight_offset;
        }
        float c = 1.f, s = 0.f;
        if (rotate) {
            c = cos_tab[(int64_t)pos * half + i];
            s = sin_tab[(int64_t)pos * half + i];
        }
        out[i] = from_float<TA>(a * c - b * s);
        out[i + half] = from_float<TA>(a * s + b * c);
    }
    // Pass-through part beyond the rotated width (everything when nothing rotates: rot_dim is 0 then).
    for (int i = 2 * half + lane; i < Dh; i += 32) {
        float a = to_float(x[i]) * inv;
        if (nw) a *= to_float(nw[i]) + weight_offset;
        out[i] = from_float<TA>(a);
    }
}

// The same for bfloat16 activations with 4-byte and 8-byte accesses: lane l holds the pairs
// (2l, 2l+1) of both rotary halves (and the next 64 for head sizes above 128), so a warp reads a head's
// row in whole 128-byte lines.  Needs rot_dim % 4 == 0, rot_dim <= 256, Dh % 4 == 0, row_stride % 4 == 0.
template <typename TW>
__global__ void qk_norm_rope_kv_vec_kernel(
    __nv_bfloat16* __restrict__ qkv, int64_t row_stride, int Hq, int Hkv, int Dh,
    const TW* __restrict__ q_norm_w, const TW* __restrict__ k_norm_w, float eps, float weight_offset,
    const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int rot_dim, int max_pos,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token,
    const int* __restrict__ block_table, int bt_stride, int n_seqs,
    __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, int page_size, int num_pages,
    int n_tokens, int* status) {
    pdl_wait();
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    const int unit = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int heads_per_token = Hq + 2 * Hkv;
    if (unit >= n_tokens * heads_per_token) return;
    const int t = unit / heads_per_token;
    const int hh = unit - t * heads_per_token;
    const int pos = positions[t];
    __nv_bfloat16* x = qkv + (int64_t)t * row_stride + (int64_t)hh * Dh;
    const bool is_q = hh < Hq;
    const bool is_k = !is_q && hh < Hq + Hkv;
    const int kv_head = is_q ? 0 : (is_k ? hh - Hq : hh - Hq - Hkv);

    __nv_bfloat16* dst = nullptr;
    if (!is_q) {
        __nv_bfloat16* cache = is_k ? k_cache : v_cache;
        if (cache == nullptr) {
            if (!is_k) return;
        } else {
            const int seq = seq_of_token[t];
            if (seq < 0 || seq >= n_seqs) {
                if (lane == 0) imp_report(status, IMP_BAD_SEQUENCE);
                return;
            }
            const int slot_page = pos / page_size;
            if (pos < 0 || slot_page >= bt_stride) {
                if (lane == 0) imp_report(status, IMP_TAGGED(IMP_BAD_POSITION, 6));
                return;
            }
            const int page = block_table[(int64_t)seq * bt_stride + slot_page];
            if (page < 0 || page >= num_pages) {
                if (lane == 0) imp_report(status, IMP_BAD_PAGE);
                return;
            }
            dst = cache + (((int64_t)page * Hkv + kv_head) * page_size + (pos - slot_page * page_size)) * Dh;
        }
    }
    if (!is_q && !is_k) {  // v: plain copy into its page, 8 bytes per lane
        for (int i = lane * 4; i < Dh; i += 128) *reinterpret_cast<uint2*>(dst + i) = *reinterpret_cast<const uint2*>(x + i);
        return;
    }
    const TW* nw = is_q ? q_norm_w : k_norm_w;
    const int half = rot_dim >> 1;
    const bool rotate = cos_tab != nullptr && half > 0;
    if (rotate && (pos < 0 || pos >= max_pos)) {
        if (lane == 0) imp_report(status, IMP_TAGGED(IMP_BAD_POSITION, 6));
        return;
    }
    // pairs j = lane, lane + 32 of each half (half <= 128 elements = 64 pairs)
    float2 a[2], b[2];
    float ss = 0.f;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        a[r] = b[r] = make_float2(0.f, 0.f);
        if (2 * j < half) {
            a[r] = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(x)[j]);
            b[r] = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(x + half)[j]);
            ss += a[r].x * a[r].x + a[r].y * a[r].y + b[r].x * b[r].x + b[r].y * b[r].y;
        }
    }
    for (int i = 2 * half + lane; i < Dh; i += 32) {   // the part beyond the rotated width
        const float v = __bfloat162float(x[i]);
        ss += v * v;
    }
    float inv = 1.f;
    if (nw) inv = rsqrtf(warp_sum(ss) / (float)Dh + eps);
    __nv_bfloat16* out = is_q ? x : (dst ? dst : x);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = lane + 32 * r;
        if (2 * j >= half) continue;
        float2 av = make_float2(a[r].x * inv, a[r].y * inv), bv = make_float2(b[r].x * inv, b[r].y * inv);
        if (nw) {
            av.x *= to_float(nw[2 * j]) + weight_offset;
            av.y *= to_float(nw[2 * j + 1]) + weight_offset;
            bv.x *= to_float(nw[2 * j + half]) + weight_offset;
            bv.y *= to_float(nw[2 * j + 1 + half]) + weight_offset;
        }
        float2 c = make_float2(1.f, 1.f), sn = make_float2(0.f, 0.f);
        if (rotate) {
            c = *reinterpret_cast<const float2*>(cos_tab + (int64_t)pos * half + 2 * j);
            sn = *reinterpret_cast<const float2*>(sin_tab + (int64_t)pos * half + 2 * j);
        }
        reinterpret_cast<__nv_bfloat162*>(out)[j] = __floats2bfloat162_rn(av.x * c.x - bv.x * sn.x, av.y * c.y - bv.y * sn.y);
        reinterpret_cast<__nv_bfloat162*>(out + half)[j] =
            __floats2bfloat162_rn(av.x * sn.x + bv.x * c.x, av.y * sn.y + bv.y * c.y);
    }
    for (int i = 2 * half + lane; i < Dh; i += 32) {
        float v = __bfloat162float(x[i]) * inv;
        if (nw) v *= to_float(nw[i]) + weight_offset;
        out[i] = __float2bfloat16_rn(v);
    }
}

// The same for heads of 64 or 128 that rotate over their whole width, in 16-byte pieces: DH / 8 lanes a head, lane l of a head
// with dimensions 8 l ... 8 l + 7, a warp with eight (sixteen) heads of one token whose rows are asked for together and whose
// table entries and norm weights are read once.  A dimension's partner is half a head, DH / 16 lanes, away.
// It stands behind the plain product where that is faster than the fused one (256 tokens and more), and gives that one's bits.
// What bounds it: the rows' way in and out.  32 + 8 + 8 heads of 128: 512 tokens 6.1 us, 2,048 17.5; a warp per head with 4-byte
// pieces and the tables read for every head 8.8 and 28.3.
template <int DH, typename TW>
__global__ void __launch_bounds__(128) qk_norm_rope_kv_heads_kernel(
    __nv_bfloat16* __restrict__ qkv, int64_t row_stride, int Hq, int Hkv, const TW* __restrict__ q_norm_w, const TW* __restrict__ k_norm_w,
    float eps, float weight_offset, const float* __restrict__ cos_tab, const float* __restrict__ sin_tab, int max_pos,
    const int* __restrict__ positions, const int* __restrict__ seq_of_token, const int* __restrict__ block_table, int bt_stride, int n_seqs,
    __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache, int page_size, int num_pages, int n_tokens, int* status) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int LANES = DH / 8, AT_ONCE = 32 / LANES, ROUNDS = 4, HEADS = AT_ONCE * ROUNDS, WARPS = 4;
    __shared__ uint4 rows_s[WARPS * HEADS][LANES + 1];     // padded: 16-byte reads down a column miss each other's banks
    __shared__ float inv_s[WARPS * HEADS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, heads = Hq + 2 * Hkv, chunks = (heads + HEADS - 1) / HEADS;
    const int64_t unit = (int64_t)blockIdx.x * WARPS + warp;
    const bool active = unit < (int64_t)n_tokens * chunks;   // a warp beyond the last unit only meets the others at the barriers
    const int t = active ? (int)(unit / chunks) : 0, first = active ? (int)(unit - (int64_t)t * chunks) * HEADS + lane / LANES : heads;
    const int piece = (lane % LANES) * 8, pair = piece % (DH / 2);   // the lane's dimensions, and their place in the tables
    const bool upper = piece >= DH / 2;
    __nv_bfloat16* row = qkv + (int64_t)t * row_stride + piece;
    uint4 raw[ROUNDS];
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
        const int hh = first + i * AT_ONCE;
        raw[i] = hh < heads ? *reinterpret_cast<const uint4*>(row + (int64_t)hh * DH) : make_uint4(0u, 0u, 0u, 0u);
    }
    const int pos = positions[t];
    const bool in_table = pos >= 0 && pos < max_pos;
    float co[8], si[8];
    if (in_table) {
#pragma unroll
        for (int e = 0; e < 8; e += 4) {
            const float4 c4 = *reinterpret_cast<const float4*>(cos_tab + (int64_t)pos * (DH / 2) + pair + e);
            const float4 s4 = *reinterpret_cast<const float4*>(sin_tab + (int64_t)pos * (DH / 2) + pair + e);
            co[e] = c4.x, co[e + 1] = c4.y, co[e + 2] = c4.z, co[e + 3] = c4.w;
            si[e] = s4.x, si[e + 1] = s4.y, si[e + 2] = s4.z, si[e + 3] = s4.w;
        }
    }
    int64_t place = -1;                    // of the token in a kv head's pages
    int fault = 0;
    if (k_cache) {
        const int seq = seq_of_token[t], slot_page = pos / page_size;
        if (seq < 0 || seq >= n_seqs) fault = IMP_BAD_SEQUENCE;
        else if (pos < 0 || slot_page >= bt_stride) fault = IMP_TAGGED(IMP_BAD_POSITION, 6);
        else {
            const int page = block_table[(int64_t)seq * bt_stride + slot_page];
            if (page < 0 || page >= num_pages) fault = IMP_BAD_PAGE;
            else place = (int64_t)page * Hkv * page_size + (pos - slot_page * page_size);
        }
    }
    const bool norm = q_norm_w != nullptr;
    float inv[ROUNDS] = {1.f, 1.f, 1.f, 1.f};
    if (norm) {
        // One chain over a head in the order of its dimensions, as the fused epilogue's thread adds them, which holds a whole
        // head: here a thread a head, for the CTA's heads at once.
#pragma unroll
        for (int i = 0; i < ROUNDS; ++i) rows_s[warp * HEADS + i * AT_ONCE + lane / LANES][lane % LANES] = raw[i];
        __syncthreads();
        if (threadIdx.x < WARPS * HEADS) {
            float ss = 0.f;
#pragma unroll
            for (int p = 0; p < LANES; ++p) {
                const uint4 u = rows_s[threadIdx.x][p];
                const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(v[e]);
                    ss = fmaf(f.x, f.x, ss);
                    ss = fmaf(f.y, f.y, ss);
                }
            }
            inv_s[threadIdx.x] = rsqrtf(ss / (float)DH + eps);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ROUNDS; ++i) inv[i] = inv_s[warp * HEADS + i * AT_ONCE + lane / LANES];
    }
    if (!active) return;
#pragma unroll
    for (int i = 0; i < ROUNDS; ++i) {
        const int hh = first + i * AT_ONCE;
        const bool is_q = hh < Hq, is_k = !is_q && hh < Hq + Hkv, there = hh < heads;
        __nv_bfloat16* dst = row + (int64_t)hh * DH;
        bool write = there;
        if (there && !is_q) {
            if (k_cache) {
                const int kv = is_k ? hh - Hq : hh - Hq - Hkv;
                if (fault) imp_report(status, fault);
                write = fault == 0;
                dst = (is_k ? k_cache : v_cache) + (place + (int64_t)kv * page_size) * DH + piece;
            } else {
                write = is_k;
            }
        }
        if (there && (is_q || is_k) && !in_table) {
            if (write) imp_report(status, IMP_TAGGED(IMP_BAD_POSITION, 6));
            write = false;
        }
        if (there && !is_q && !is_k && write) *reinterpret_cast<uint4*>(dst) = raw[i];
        // all lanes take part in the exchanges; lanes beyond the last head work on zeros
        const __nv_bfloat162* in = reinterpret_cast<const __nv_bfloat162*>(&raw[i]);
        float x[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(in[e]);
            x[2 * e] = f.x, x[2 * e + 1] = f.y;
        }
        if (norm) {
            const TW* nw = is_q ? q_norm_w : k_norm_w;
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = x[e] * inv[i] * (to_float(nw[piece + e]) + weight_offset);
        }
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = __shfl_xor_sync(0xffffffffu, x[e], LANES / 2);
        if (write && (is_q || is_k)) {
            uint4 out;
            __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float r[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int k = 2 * e + j;
                    r[j] = upper ? y[k] * si[k] + x[k] * co[k] : x[k] * co[k] - y[k] * si[k];
                }
                o2[e] = __floats2bfloat162_rn(r[0], r[1]);
            }
            *reinterpret_cast<uint4*>(dst) = out;
        }
    }
}

// qkv: [n_tokens, row_stride] with q heads, then k heads, then v heads, each head_dim wide.
// q is normalised and rotated in place; k (normalised, rotated) and v go to the pages
// (when k_cache/v_cache are null, k is rotated in place and v is left alone).
IMP_API int imp_qk_norm_rope_kv_write(
    void* qkv, int64_t row_stride, int n_tokens, int Hq, int Hkv, int Dh,
    const void* q_norm_w, const void* k_norm_w, float eps, float weight_offset, int w_dtype,
    const float* cos_tab, const float* sin_tab, int rot_dim, int max_pos,
    const int* positions, const int* seq_of_token, const int* block_table, int bt_stride, int n_seqs,
    void* k_cache, void* v_cache, int page_size, int num_pages, int act_dtype, int* status, void* stream) {
    if (n_tokens == 0) return 0;
    IMP_CHECK_ARG(qkv && positions && Hq >= 0 && Hkv >= 0 && Dh > 0, "imp_qk_norm_rope_kv_write: bad argument");
    IMP_CHECK_ARG(rot_dim >= 0 && rot_dim <= Dh && rot_dim % 2 == 0,
                  "imp_qk_norm_rope_kv_write: rotary width %d must be even and at most head_dim %d", rot_dim, Dh);
    IMP_CHECK_ARG((k_cache == nullptr) == (v_cache == nullptr), "imp_qk_norm_rope_kv_write: k and v cache must both be set or both be null");
    if (k_cache) IMP_CHECK_ARG(seq_of_token && block_table && page_size > 0 && num_pages > 0,
                               "imp_qk_norm_rope_kv_write: cache write needs the batch's block table");
    IMP_CHECK_ARG((q_norm_w == nullptr) == (k_norm_w == nullptr), "imp_qk_norm_rope_kv_write: q and k norm weights must both be set or both be null");
    cudaStream_t s = (cudaStream_t)stream;
    const int warps = 4;
    const int64_t units = (int64_t)n_tokens * (Hq + 2 * Hkv);
    const int grid = (int)((units + warps - 1) / warps);
    if (cos_tab == nullptr) rot_dim = 0;
#define LAUNCH(TA, TW)                                                                                      \
    imp_launch(qk_norm_rope_kv_kernel<TA, TW>, dim3(grid), dim3(warps * 32), 0, s,                          \
        (TA*)qkv, row_stride, Hq, Hkv, Dh, (const TW*)q_norm_w, (const TW*)k_norm_w, eps, weight_offset,    \
        cos_tab, sin_tab, rot_dim, max_pos, positions, seq_of_token, block_table, bt_stride, n_seqs,        \
        (TA*)k_cache, (TA*)v_cache, page_size, num_pages, n_tokens, status)
    const bool vec = act_dtype == IMP_BF16 && rot_dim % 4 == 0 && rot_dim <= 256 && Dh % 4 == 0 && row_stride % 4 == 0 &&
                     (uintptr_t)qkv % 8 == 0 && (uintptr_t)k_cache % 8 == 0 && (uintptr_t)v_cache % 8 == 0 &&
                     (uintptr_t)cos_tab % 8 == 0 && (uintptr_t)sin_tab % 8 == 0;
#define LAUNCH_VEC(TW)                                                                                      \
    imp_launch(qk_norm_rope_kv_vec_kernel<TW>, dim3(grid), dim3(warps * 32), 0, s,                          \
        (__nv_bfloat16*)qkv, row_stride, Hq, Hkv, Dh, (const TW*)q_norm_w, (const TW*)k_norm_w, eps, weight_offset, \
        cos_tab, sin_tab, rot_dim, max_pos, positions, seq_of_token, block_table, bt_stride, n_seqs,        \
        (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, page_size, num_pages, n_tokens, status)
    const uintptr_t ptrs = (uintptr_t)qkv | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)cos_tab | (uintptr_t)sin_tab;
    const bool heads16 = vec && n_tokens >= 256 && (Dh == 64 || Dh == 128) && rot_dim == Dh && row_stride % 8 == 0 && ptrs % 16 == 0;
#define LAUNCH_HEADS(DH, TW)                                                                                \
    imp_launch(qk_norm_rope_kv_heads_kernel<DH, TW>,                                                        \
        dim3((unsigned)(((int64_t)n_tokens * ((Hq + 2 * Hkv + 1024 / DH - 1) / (1024 / DH)) + 3) / 4)), dim3(128), 0, s, \
        (__nv_bfloat16*)qkv, row_stride, Hq, Hkv, (const TW*)q_norm_w, (const TW*)k_norm_w, eps, weight_offset, \
        cos_tab, sin_tab, max_pos, positions, seq_of_token, block_table, bt_stride, n_seqs,                 \
        (__nv_bfloat16*)k_cache, (__nv_bfloat16*)v_cache, page_size, num_pages, n_tokens, status)
    if (heads16 && Dh == 128 && w_dtype == IMP_F32) LAUNCH_HEADS(128, float);
    else if (heads16 && Dh == 128) LAUNCH_HEADS(128, __nv_bfloat16);
    else if (heads16 && w_dtype == IMP_F32) LAUNCH_HEADS(64, float);
    else if (heads16) LAUNCH_HEADS(64, __nv_bfloat16);
    else if (vec && w_dtype == IMP_F32) LAUNCH_VEC(float);
    else if (vec) LAUNCH_VEC(__nv_bfloat16);
    else if (act_dtype == IMP_F32 && w_dtype == IMP_F32) LAUNCH(float, float);
    else if (act_dtype == IMP_F32) LAUNCH(float, __nv_bfloat16);
    else if (w_dtype == IMP_F32) LAUNCH(__nv_bfloat16, float);
    else LAUNCH(__nv_bfloat16, __nv_bfloat16);
#undef LAUNCH
#undef LAUNCH_VEC
#undef LAUNCH_HEADS
    IMP_RETURN_LAUNCH();
}
