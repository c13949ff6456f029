// The layers of a decode step in one launch (decode_stack.cu): what the host fills in.
#pragma once
#include <stdint.h>

constexpr int STACK_MAX_TOKENS = 8;     // columns of one tensor operation
constexpr int STACK_MAX_LAYERS = 128;
constexpr int STACK_SS_STRIDE = 256;    // floats between two tokens' shares of the sums of squares

struct StackLayer {
    const void *w_qkv, *w_o, *w_gu, *w_down;      // bfloat16, dense; gate and up rows alternate in runs of 8
    const float *norm1, *norm2;                   // [d]
    const float *q_norm, *k_norm;                 // [128] or both null
    void *k_pages, *v_pages;                      // bfloat16 [pages, hkv, page_size, 128]
};

struct StackArgs {
    const StackLayer* layers;   // device
    int n_layers, T, d, F, hq, hkv;
    float* h;                   // [T, d], updated
    // scratch: [T, (hq + 2 hkv) 128] | [T, hq 128] | [T, F] bfloat16; [T, STACK_SS_STRIDE]; [items, hq / hkv, 128]; [items, hq / hkv, 2]
#ifdef __CUDACC__
    __nv_bfloat16 *qkv, *attn, *hid;
#else
    void *qkv, *attn, *hid;
#endif
    float *ss, *part_o, *part_ml;
    unsigned* sync;             // [2 + T hkv], zero between launches
    const int *positions, *seq_of_token, *block_table;
    int bt_stride, n_seqs, page_size, num_pages;
    const float *cos_tab, *sin_tab;   // [max_pos, 64]
    int max_pos;
    float eps1, eps2, qk_eps, scale_log2;
    int act;                    // GateAct's kinds, without a bias
    float act_limit;
    int* status;
    int n_stages, scratch_at, ring_at;    // filled in by the launcher
};
