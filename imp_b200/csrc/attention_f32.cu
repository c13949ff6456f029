// Paged attention of the float32 path for head sizes 64, 128 and 256, without a score bias or a sink (those, and other head
// sizes, stay with the plain kernel of attention_generic.cu).
//
// One order of operations per (token, query head), fixed by the token's position alone: keys in chunks of 32 (chunk c holds
// positions 32 c ... 32 c + 31); a chunk's scores, maximum, sum of exponentials and weighted values are found on their own
// and then merged, chunks ascending.  So the result is the same bits whatever else is in the batch, however the prompt was
// cut, and whichever of the two forms computed it:
//   a warp a token   (many tokens): eight neighbouring tokens a CTA, which mostly walk the same keys and meet them in L1.
//   a CTA a token    (few tokens): its warps take a chunk each, the merge follows in order through shared memory.
// A warp serves one or two query heads of a kv head; with two, a key and a value are read once for both.  A lane holds Dh / 32
// neighbouring entries: rows of K and V are read whole (512 bytes an instruction at head size 128), and the 32 dot products
// of a chunk are summed over the lanes by one transposing tree of 31 exchanges that leaves key i's score in lane i.
//
// What bounds it: latency at one row a sequence, the instructions' issue at many.  16 query heads over 8 kv heads of 128:
//   four sequences of 60 to 260 keys, a token each     8.1 us with 16 warps of one head, 11.3 with 8 of two, 10.3 with 8 of one
//   sixteen of 300                                     16.0, 13.1, 22.5
//   four prompts of 60 to 260 tokens (a warp a token)  82 us with two heads and two CTAs an SM, 101 with one CTA, 89 with one head
// hence the lines in af_launch.  The plain kernel (a thread a row of K, the values of 128 keys in one chain) took 24 ms where
// this one takes 4.5: 28 layers, eight steps of four single tokens and a step of 580 tokens.
#include "common.cuh"
#include "attention_f32.h"

namespace {

constexpr int AF_KEYS = 32;

struct AfArgs {
    float* out;
    const float *q, *k_cache, *v_cache;
    const int *block_table, *seq_of_token, *positions;
    int* status;
    int64_t out_stride, q_stride;
    int bt_stride, n_tokens, n_seqs, Hq, Hkv, page_size, num_pages, window;
    float scale;
};

template <int DV> struct AfVec {   // Dh / 32 neighbouring floats
    float v[DV];
    __device__ __forceinline__ void load(const float* p) {
        if (DV == 2) {
            const float2 t = *(const float2*)p;
            v[0] = t.x; v[1] = t.y;
        } else {
#pragma unroll
            for (int i = 0; i < DV; i += 4) {
                const float4 t = *(const float4*)(p + i);
                v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
            }
        }
    }
    __device__ __forceinline__ void store(float* p) const {
        if (DV == 2) *(float2*)p = make_float2(v[0], v[1]);
        else
#pragma unroll
            for (int i = 0; i < DV; i += 4) *(float4*)(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    }
};

// One chunk for GH heads: maximum, sum and (this lane's) weighted values of the keys lo ... pos among j0 ... j0 + 31.
template <int DV, int GH>
__device__ __forceinline__ void af_chunk(const AfArgs& a, const AfVec<DV> (&q)[GH], const int* bt, int hk, int j0, int lo, int pos,
                                         int64_t* offs, float (&m)[GH], float (&l)[GH], AfVec<DV> (&acc)[GH]) {
    const int lane = threadIdx.x & 31, j = j0 + lane;
    int64_t off = -1;
    if (j >= lo && j <= pos) {
        const int page = bt[j / a.page_size];
        if (page < 0 || page >= a.num_pages) imp_report(a.status, IMP_BAD_PAGE);
        else off = (((int64_t)page * a.Hkv + hk) * a.page_size + j % a.page_size) * (32 * DV);
    }
    __syncwarp();
    offs[lane] = off;
    __syncwarp();
    float dot[GH][AF_KEYS];
#pragma unroll
    for (int i = 0; i < AF_KEYS; ++i) {
        const int64_t o = offs[i];
        AfVec<DV> k;
        if (o >= 0) k.load(a.k_cache + o + lane * DV);
        else
#pragma unroll
            for (int d = 0; d < DV; ++d) k.v[d] = 0.f;
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            float s = __fmul_rn(q[g].v[0], k.v[0]);
#pragma unroll
            for (int d = 1; d < DV; ++d) s = __fmaf_rn(q[g].v[d], k.v[d], s);
            dot[g][i] = s;
        }
    }
    float p[GH];
#pragma unroll
    for (int g = 0; g < GH; ++g) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float keep = up ? dot[g][i + o] : dot[g][i], give = up ? dot[g][i] : dot[g][i + o];
                dot[g][i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, o));
            }
        }
        const float s = off >= 0 ? __fmul_rn(dot[g][0], a.scale) : -INFINITY;
        m[g] = warp_max(s);
        p[g] = s == -INFINITY ? 0.f : expf(__fsub_rn(s, m[g]));
        l[g] = warp_sum(p[g]);
#pragma unroll
        for (int d = 0; d < DV; ++d) acc[g].v[d] = 0.f;
    }
#pragma unroll 8
    for (int i = 0; i < AF_KEYS; ++i) {
        const int64_t o = offs[i];
        AfVec<DV> v;
        if (o >= 0) v.load(a.v_cache + o + lane * DV);
        else
#pragma unroll
            for (int d = 0; d < DV; ++d) v.v[d] = 0.f;
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            const float w = __shfl_sync(0xffffffffu, p[g], i);
#pragma unroll
            for (int d = 0; d < DV; ++d) acc[g].v[d] = __fmaf_rn(w, v.v[d], acc[g].v[d]);
        }
    }
}

// (m, l) of what was merged so far <- with a chunk's; the factors of the two accumulators come back.
__device__ __forceinline__ void af_merge(float& m, float& l, float cm, float cl, float& old_f, float& new_f) {
    const float top = fmaxf(m, cm);
    old_f = m == -INFINITY ? 0.f : expf(__fsub_rn(m, top));
    new_f = cm == -INFINITY ? 0.f : expf(__fsub_rn(cm, top));
    l = __fmaf_rn(l, old_f, __fmul_rn(cl, new_f));
    m = top;
}
__device__ __forceinline__ float af_blend(float acc, float old_f, float c, float new_f) { return __fmaf_rn(acc, old_f, __fmul_rn(c, new_f)); }
// Without a key that counts the result is 0 where the token's own page is missing, and no number where every score is -inf.
__device__ __forceinline__ float af_over(float acc, float l, bool own) {
    return l > 0.f ? __fmul_rn(acc, __fdiv_rn(1.f, l)) : l == 0.f && !own ? 0.f : __int_as_float(0x7fffffff);
}

// Grid (tokens / 8 or tokens, kv heads x groups of GH query heads).
template <int DV, int GH, int AF_WARPS, int MIN_CTAS, bool CTA_A_TOKEN>
__global__ void __launch_bounds__(AF_WARPS * 32, MIN_CTAS) attention_f32_kernel(const AfArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    constexpr int DH = 32 * DV;
    __shared__ int64_t offs[AF_WARPS][AF_KEYS];
    __shared__ __align__(16) float part[CTA_A_TOKEN ? AF_WARPS * GH * DH : 4];   // written 16 bytes at a time
    __shared__ float part_m[AF_WARPS][GH], part_l[AF_WARPS][GH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = a.Hq / a.Hkv, sets = (G + GH - 1) / GH, hk = blockIdx.y / sets, h0 = hk * G + blockIdx.y % sets * GH;
    const int n_heads = min(GH, (hk + 1) * G - h0);
    const int t = CTA_A_TOKEN ? blockIdx.x : blockIdx.x * AF_WARPS + warp;
    if (t >= a.n_tokens) return;   // a whole warp, and only in the form without barriers
    const int seq = a.seq_of_token[t], pos = a.positions[t];
    float* out = a.out + t * a.out_stride + (int64_t)h0 * DH;
    if (seq < 0 || seq >= a.n_seqs || pos < 0 || pos / a.page_size >= a.bt_stride) {
        if (lane == 0) imp_report(a.status, seq < 0 || seq >= a.n_seqs ? IMP_BAD_SEQUENCE : IMP_BAD_POSITION);
        if (!CTA_A_TOKEN || warp == 0)
            for (int i = lane; i < n_heads * DH; i += 32) out[i] = 0.f;
        return;
    }
    const int* bt = a.block_table + (int64_t)seq * a.bt_stride;
    const int lo = imp_first_key(pos, a.window), c0 = lo / AF_KEYS, c1 = pos / AF_KEYS;
    const int own_page = bt[pos / a.page_size];
    const bool own = own_page >= 0 && own_page < a.num_pages;
    AfVec<DV> q[GH];
#pragma unroll
    for (int g = 0; g < GH; ++g)
        q[g].load(a.q + t * a.q_stride + (int64_t)(h0 + min(g, n_heads - 1)) * DH + lane * DV);
    float cm[GH], cl[GH];
    AfVec<DV> cacc[GH];
    if (!CTA_A_TOKEN) {
        float m[GH], l[GH];
        AfVec<DV> acc[GH];
#pragma unroll
        for (int g = 0; g < GH; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.f;
#pragma unroll
            for (int d = 0; d < DV; ++d) acc[g].v[d] = 0.f;
        }
        for (int c = c0; c <= c1; ++c) {
            af_chunk<DV, GH>(a, q, bt, hk, c * AF_KEYS, lo, pos, offs[warp], cm, cl, cacc);
#pragma unroll
            for (int g = 0; g < GH; ++g) {
                float fo, fn;
                af_merge(m[g], l[g], cm[g], cl[g], fo, fn);
#pragma unroll
                for (int d = 0; d < DV; ++d) acc[g].v[d] = af_blend(acc[g].v[d], fo, cacc[g].v[d], fn);
            }
        }
#pragma unroll
        for (int g = 0; g < GH; ++g) {
#pragma unroll
            for (int d = 0; d < DV; ++d) acc[g].v[d] = af_over(acc[g].v[d], l[g], own);
            if (g < n_heads) acc[g].store(out + g * DH + lane * DV);
        }
    } else {
        constexpr int MINE = (GH * DH + AF_WARPS * 32 - 1) / (AF_WARPS * 32);   // merged outputs of a thread
        float m[MINE], l[MINE], acc[MINE];
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            m[i] = -INFINITY;
            l[i] = acc[i] = 0.f;
        }
        for (int r = c0; r <= c1; r += AF_WARPS) {
            if (r + warp <= c1) {
                af_chunk<DV, GH>(a, q, bt, hk, (r + warp) * AF_KEYS, lo, pos, offs[warp], cm, cl, cacc);
#pragma unroll
                for (int g = 0; g < GH; ++g) {
                    cacc[g].store(part + (warp * GH + g) * DH + lane * DV);
                    if (lane == 0) {
                        part_m[warp][g] = cm[g];
                        part_l[warp][g] = cl[g];
                    }
                }
            }
            __syncthreads();
            const int n = min(AF_WARPS, c1 - r + 1);
#pragma unroll
            for (int i = 0; i < MINE; ++i) {
                const int e = threadIdx.x + i * AF_WARPS * 32, g = e / DH;
                if (e < GH * DH)
                    for (int w = 0; w < n; ++w) {
                        float fo, fn;
                        af_merge(m[i], l[i], part_m[w][g], part_l[w][g], fo, fn);
                        acc[i] = af_blend(acc[i], fo, part[w * GH * DH + e], fn);
                    }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
            const int e = threadIdx.x + i * AF_WARPS * 32;
            if (e < n_heads * DH) out[e] = af_over(acc[i], l[i], own);
        }
    }
}

template <int DV, int GH, int WARPS, int MIN_CTAS, bool CTA_A_TOKEN>
cudaError_t af_run(const AfArgs& a, cudaStream_t stream) {
    const int sets = (a.Hq / a.Hkv + GH - 1) / GH;
    return imp_launch(attention_f32_kernel<DV, GH, WARPS, MIN_CTAS, CTA_A_TOKEN>, dim3(CTA_A_TOKEN ? a.n_tokens : (a.n_tokens + WARPS - 1) / WARPS, a.Hkv * sets),
                      WARPS * 32, 0, stream, a);
}

template <int DV>
cudaError_t af_launch(const AfArgs& a, cudaStream_t stream) {
    const int64_t heads = (int64_t)a.n_tokens * a.Hq;
    if (heads <= imp_sm_count()) return af_run<DV, 1, 16, 1, true>(a, stream);
    if (a.Hq == a.Hkv) return heads <= 8ll * imp_sm_count() ? af_run<DV, 1, 8, 1, true>(a, stream) : af_run<DV, 1, 8, 3, false>(a, stream);
    return heads <= 8ll * imp_sm_count() ? af_run<DV, 2, 8, 1, true>(a, stream) : af_run<DV, 2, 8, 2, false>(a, stream);
}

}  // namespace

int imp_attention_f32(float* out, int64_t out_stride, const float* q, int64_t q_stride, const float* k_cache, const float* v_cache,
                      const int* block_table, int bt_stride, const int* seq_of_token, const int* positions, int n_tokens, int n_seqs,
                      int Hq, int Hkv, int Dh, int page_size, int num_pages, float scale, int window, int* status, cudaStream_t stream) {
    const uintptr_t ptrs = (uintptr_t)out | (uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache;
    if ((Dh != 64 && Dh != 128 && Dh != 256) || ptrs % 16 || out_stride % 4 || q_stride % 4 || Hq > 65535) return IMP_ERR_UNSUPPORTED;
    const AfArgs a{out, q, k_cache, v_cache, block_table, seq_of_token, positions, status, out_stride, q_stride,
                   bt_stride, n_tokens, n_seqs, Hq, Hkv, page_size, num_pages, window, scale};
    const cudaError_t e = Dh == 64 ? af_launch<2>(a, stream) : Dh == 128 ? af_launch<4>(a, stream) : af_launch<8>(a, stream);
    if (e != cudaSuccess) {
        imp_set_error("imp_attention_f32: %s", cudaGetErrorString(e));
        return (int)e;
    }
    IMP_RETURN_LAUNCH();
}
