// Interface of the token-N kernels (moe_tokn.cu) to the launchers in moe_bf16.cu and moe_mxfp8.cu.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace pmoe {

struct ToknProblem {
    const void *x, *w, *w2;
    void *out;
    const int32_t *sorted_ids, *expert_ids, *npp;
    const float *topk_weights;
    const int32_t *live_rows;   // optional, as in CallExtras
    void *gu_out;               // optional, as in CallExtras
    int top_k, M, K, N, E, sorted_num, bpc;
    // mxfp8 operands if w_scales is set: the caller's scales (x_scales 4-byte aligned) and the workspace regions of the
    // rows' and the activations' scale tiles, sorted_num * K / 32 and sorted_num * N / 64 bytes
    const void *x_scales, *w_scales, *w2_scales;
    uint8_t *x_sf, *act_sf;
};

// bytes of the work-item list and the per-row tokens and weights for a routing table of `sorted_num` rows (16-byte aligned region)
size_t tokn_items_bytes(int sorted_num);

// rows of one work item at most, for `rows` routed rows over E experts
int tokn_cap(long long rows, int E, bool mx);

// act [sorted_num, N/2] (bf16 or e4m3) and items are regions of the call's workspace; `phases` as in phase_mask()
int run_tokn(const ToknProblem &p, void *act, void *items, int phases, cudaStream_t stream);

// Row-space GEMMs of the bf16 backward pass on the same kernel. The 128-row blocks that hold routed rows as block * 1024 +
// expert, their number, and one past every expert's last routed row, all on the device.
struct ToknBlocks {
    const int32_t *blocks, *count, *row_end;
};
// gate_up: gu = xs . W1^T; d_act: dgu, actw, dwt from dos . W2 and gu; d_xs: dxs = dgu . W1. Written are the blocks' rows up to
// the expert's last routed one, rounded up to 32; zeros in dgu and actw for the padding rows among them.
struct ToknBackward {
    const void *xs, *w1, *w2, *dos;
    void *gu, *dgu, *actw, *dxs;
    float *dwt;                 // d_topk_weights, zeroed before, or null
    const int32_t *sorted_ids;
    const float *topk_weights;
    ToknBlocks list;
    int top_k, M, K, N, E, sorted_num;
};
enum class ToknStep { gate_up, d_act, d_xs };
int tokn_block_gemm(const ToknBackward &p, ToknStep step, cudaStream_t stream);

}  // namespace pmoe
