// Routed experts with many rows per expert (prefill-sized batches): the whole layer up to the combine.
//
// With single blocks of eight rows the grouped GEMM streams and decodes an expert's matrices once per eight routed rows, which is right
// for decode batches and wasteful once experts see tens of rows.  The reference answers that by growing its moe block from 8 to 64
// rows with T * top_k / E (cuda/src/sglang_exl3/kernels/marlin_moe.py:52-57 of 0xSero/trellis-serve); here the routing stays aligned to
// eight rows and the align kernel lists items of up to 128 consecutive rows of one expert, which share every decoded weight:
//
//   align + items
//   gather, * suh, Had128 -> B operand               (gate and up inputs)
//   grouped GEMM gate|up                             (rotated basis, fp16)
//   Had128 * svh -> SiLU(gate) * up -> fp16 -> * suh2 -> Had128 -> B operand
//   grouped GEMM down                                (rotated basis, fp16)
//   Had128 * svh2 -> yd[slot, :]                     (the combine kernel closes the layer)
//
// Same arithmetic as the decode-sized layer (cuda/csrc/exl3_marlin_moe.cu:210-292) up to the rounding of the weights and of the
// rotated-basis products to fp16, which the dense many-row path has as well.
#include <cstring>

#include "exl3_moe_kernel.cuh"

namespace exl3 {

static inline size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

struct MoeTcLayout {
    size_t sorted, experts, counts, items, blk, xf13, gu, xf2, yd_rot, total;
    int cap;
};

static MoeTcLayout moe_tc_layout(int slots, int num_local, int hidden, int inter)
{
    MoeTcLayout l;
    const size_t used = (size_t)(slots < num_local ? slots : num_local);           // experts that can receive a slot
    l.cap = (int)(((size_t)slots + used * (MOE_BLOCK_ROWS - 1) + MOE_BLOCK_ROWS - 1) / MOE_BLOCK_ROWS * MOE_BLOCK_ROWS);
    size_t off = MOE_ERR_WORDS * 4;                                                 // header: error word
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += up256(bytes);
        return at;
    };
    const size_t blocks = (size_t)l.cap / MOE_BLOCK_ROWS + 1;
    l.sorted = take((size_t)l.cap * 4);
    l.experts = take(blocks * 4);
    l.counts = take(16);                                                            // rows, items, rows of the largest item
    l.items = take(blocks * sizeof(int4));
    l.blk = take(blocks * sizeof(int2));
    l.xf13 = take((size_t)2 * l.cap * hidden * 2);
    l.gu = take((size_t)l.cap * 2 * inter * 2);
    l.xf2 = take((size_t)l.cap * inter * 2);
    l.yd_rot = take((size_t)l.cap * hidden * 2);
    l.total = off;
    return l;
}

size_t moe_tc_workspace_bytes(int slots, int num_local, int hidden, int inter)
{
    return moe_tc_layout(slots, num_local, hidden, inter).total;
}

int launch_moe_tc_experts(const void* x, int x_bf16, int top_k, int hidden, int inter, const int* topk_ids, int slots, int num_experts,
                          const int* expert_map, int num_local, const uint32_t* w13, const __half* suh13, const __half* svh13,
                          const uint32_t* w2, const __half* suh2, const __half* svh2, int K, int codebook, __half* yd, unsigned char* ws,
                          cudaStream_t st, const float* weights, int* place, int y_bf16)
{
    constexpr int MODE = GEMV_PAIRED;
    const MoeTcLayout w = moe_tc_layout(slots, num_local, hidden, inter);
    int* sorted_ids = reinterpret_cast<int*>(ws + w.sorted);
    int* expert_ids = reinterpret_cast<int*>(ws + w.experts);
    int* counts = reinterpret_cast<int*>(ws + w.counts);
    int4* items = reinterpret_cast<int4*>(ws + w.items);
    int2* blk = reinterpret_cast<int2*>(ws + w.blk);
    __half* gu = reinterpret_cast<__half*>(ws + w.gu);
    __half* yd_rot = reinterpret_cast<__half*>(ws + w.yd_rot);

    MoeGemmLaunch l;
    memset(&l, 0, sizeof(l));
    l.sorted_ids = sorted_ids;
    l.expert_ids = expert_ids;
    l.items = items;
    l.counts = counts;
    l.err = reinterpret_cast<int*>(ws);
    l.numel = slots;
    l.rotated = 1;

    if (int rc = launch_moe_align(topk_ids, slots, num_local, MOE_BLOCK_ROWS, w.cap, sorted_ids, expert_ids, counts, expert_map,
                                  expert_map ? num_experts : 0, MOE_TC_BLOCK_ROWS / MOE_BLOCK_ROWS, items, blk, l.err, st, place))
        return rc;
    const long long stride = (long long)w.cap * hidden * 2;
    if (int rc = launch_moe_had_in_items(x, x_bf16, suh13, hidden, top_k, slots, w.cap, sorted_ids, expert_ids, counts, blk, ws + w.xf13, stride, st))
        return rc;
    l.packed = w13;
    l.expert_stride = (long long)hidden * 2 * inter * K / 32;
    l.xf = ws + w.xf13;
    l.xf_shard_stride = stride;
    l.out = gu;
    l.KG = hidden / 128;
    l.NB = 2 * inter / 128;
    l.n_total = 2 * inter;
    l.shard_end_block = inter / 128;
    if (int rc = launch_moe_gemm(l, K, codebook, MODE, st)) return rc;
    if (int rc = launch_moe_mid_items(gu, svh13, suh2, inter, slots, w.cap, sorted_ids, expert_ids, counts, blk, ws + w.xf2, st)) return rc;
    l.packed = w2;
    l.expert_stride = (long long)inter * hidden * K / 32;
    l.xf = ws + w.xf2;
    l.xf_shard_stride = 0;
    l.out = yd_rot;
    l.KG = inter / 128;
    l.NB = hidden / 128;
    l.n_total = hidden;
    l.shard_end_block = l.NB;
    if (int rc = launch_moe_gemm(l, K, codebook, MODE, st)) return rc;
    if (weights) return launch_moe_out_combine(yd_rot, svh2, weights, place, expert_ids, blk, slots / top_k, top_k, hidden, yd, y_bf16, st);
    return launch_moe_out_items(yd_rot, svh2, hidden, slots, w.cap, sorted_ids, expert_ids, counts, blk, yd, st);
}

}  // namespace exl3
