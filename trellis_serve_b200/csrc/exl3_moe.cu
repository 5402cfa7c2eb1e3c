// MoE layer pieces around the grouped GEMV (sm_100a): routing alignment, per-slot input rotations, SiLU-gated
// rotation for the down projection, router-weighted combine.  One MoE layer is
//   align -> had_in (gather, per-expert suh, gate and up) -> grouped GEMV gate|up -> glu_had_in -> grouped GEMV down -> combine
// the five-launch structure of cuda/src/sglang_exl3/kernels/marlin_moe.py:272-294 of 0xSero/trellis-serve, whose kernels
// are cuda/csrc/exl3_marlin_moe.cu:210-292 (per-slot transforms, combine) and :542-594 (decode-size align).
#include "exl3_moe_kernel.cuh"

namespace exl3 {

// ------------------------------------------------------------------------------------------------ align

// One cluster of CL CTAs.  Slots (token, k) are grouped by expert into blocks of `block` rows: sorted_ids holds the slot of every
// row (numel = padding), expert_ids the expert of every block, num_post the padded row count.  Ids outside
// [0, E) are dropped.  The order of slots inside an expert is not specified (rows are independent).
// With expert_map (int [E_global]: global id -> id in [0, E), or -1) the ids are translated first, so one class of a
// mixed-bitrate expert set gets the blocks of its own slots only, with local expert ids.
// With `items`: every expert's rows are also cut into items of up to item_blocks blocks of eight rows; items[i] = (expert, first block,
// blocks, 0), blk[b] = (first block of the item of block b, its blocks), num_post[1] = items, num_post[2] = rows of the largest one; and
// the workspace's header (error word) is cleared.  place (or null): the row of every slot, -1 for dropped ones.  Bound by latency and by shared-memory
// atomics: a CTA counts its share of the slots, reads the other CTAs' counts through distributed shared memory and lays out the experts
// itself; KEEP slots per thread are requested together and, if that takes them all, stay in registers with their rank from the
// counting (16384 slots, 256 experts: 24 us in one CTA with two passes of loads and atomics, 20 with one).
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(1024) moe_align_kernel(const int* __restrict__ topk_ids, int numel, int E, int block, int cap, int* __restrict__ sorted_ids,
                                 int* __restrict__ expert_ids, int* __restrict__ num_post, const int* __restrict__ expert_map,
                                 int E_global, int item_blocks, int4* __restrict__ items, int2* __restrict__ blk, int* __restrict__ header,
                                 int* __restrict__ place)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    extern __shared__ int sh[];
    int* count = sh;              // [E]
    int* offset = sh + E;         // [E + 1]
    int* fill = sh + 2 * E + 1;   // [E]
    constexpr int KEEP = 2;
    const int rank_cta = blockIdx.x, threads = CL * blockDim.x, thread = rank_cta * blockDim.x + threadIdx.x;      // of the cluster
    const bool one = numel <= KEEP * threads;
    int e_of[KEEP], rank[KEEP];
    auto load_ids = [&](int i0) {                       // experts of slots i0 + thread + j * threads, -1 outside [0, E)
#pragma unroll
        for (int j = 0; j < KEEP; j++) {
            const int i = i0 + thread + j * threads;
            e_of[j] = i < numel ? topk_ids[i] : -1;
        }
        if (expert_map) {
#pragma unroll
            for (int j = 0; j < KEEP; j++) e_of[j] = e_of[j] >= 0 && e_of[j] < E_global ? expert_map[e_of[j]] : -1;
        }
#pragma unroll
        for (int j = 0; j < KEEP; j++)
            if (e_of[j] >= E) e_of[j] = -1;
    };
    load_ids(0);
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        count[e] = 0;
        fill[e] = 0;
    }
    if (items && rank_cta == 0)
        for (int i = threadIdx.x; i < MOE_ERR_WORDS; i += blockDim.x) header[i] = 0;
    __syncthreads();
    for (int i0 = 0; i0 < numel; i0 += KEEP * threads) {
        if (i0 > 0) load_ids(i0);
#pragma unroll
        for (int j = 0; j < KEEP; j++) rank[j] = e_of[j] >= 0 ? atomicAdd(&count[e_of[j]], 1) : 0;
    }
    int* before = fill + E;       // CL > 1: [E], slots of the CTAs ahead; count becomes the total
    if constexpr (CL > 1) {
        ptx::cluster_sync_all();
        int sums[2] = {0, 0};
        auto gather = [&](int e) {
            sums[0] = sums[1] = 0;
            int c[CL];
#pragma unroll
            for (int r = 0; r < CL; r++) c[r] = ptx::ld_shared_cluster_s32(&count[e], r);
#pragma unroll
            for (int r = 0; r < CL; r++) {
                if (r < rank_cta) sums[0] += c[r];
                sums[1] += c[r];
            }
        };
        int total[(MOE_MAX_EXPERTS + 1023) / 1024];
#pragma unroll
        for (int i = 0; i < (MOE_MAX_EXPERTS + 1023) / 1024; i++) {
            const int e = threadIdx.x + i * 1024;
            if (e < E) {
                gather(e);
                before[e] = sums[0];
                total[i] = sums[1];
            }
        }
        ptx::cluster_sync_all();                       // every CTA has read the counts: they may change, and CTAs may leave
#pragma unroll
        for (int i = 0; i < (MOE_MAX_EXPERTS + 1023) / 1024; i++) {
            const int e = threadIdx.x + i * 1024;
            if (e < E) count[e] = total[i];
        }
    }
    // Exclusive prefix sums of the padded counts and (high word) of the items: warp scans by shuffle, warp totals through shared
    // memory; experts are taken in chunks of blockDim.x with a running carry.
    __shared__ unsigned long long warp_total[32];
    __shared__ unsigned long long carry_sh;
    __shared__ int largest;
    if (threadIdx.x == 0) {
        carry_sh = 0;
        largest = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int e0 = 0; e0 < E; e0 += blockDim.x) {
        const int e = e0 + threadIdx.x;
        const int blocks = e < E ? (count[e] + block - 1) / block : 0;
        const int n_items = items ? (blocks + item_blocks - 1) / item_blocks : 0;
        const unsigned long long own = (unsigned long long)(blocks * block) | ((unsigned long long)n_items << 32);
        unsigned long long incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += up;
        }
        if (lane == 31) warp_total[wid] = incl;
        __syncthreads();
        if (wid == 0) {
            unsigned long long t = lane < nwarps ? warp_total[lane] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long up = __shfl_up_sync(0xFFFFFFFFu, t, d);
                if (lane >= d) t += up;
            }
            warp_total[lane] = t;                      // inclusive totals of the warps
        }
        __syncthreads();
        const unsigned long long base = carry_sh + (wid > 0 ? warp_total[wid - 1] : 0);
        const unsigned long long excl = base + incl - own;
        if (e < E) {
            const int b0 = (int)(excl & 0xFFFFFFFFu) / block;
            offset[e] = b0 * block;
            if (CL == 1 || e % CL == rank_cta) {       // the CTAs share the writing
                for (int r = 0; r < blocks; r++) expert_ids[b0 + r] = e;
                for (int r = count[e]; r < blocks * block; r++) sorted_ids[b0 * block + r] = numel;
                if (items) {
                    // the expert's blocks in nearly even items
                    int at = (int)(excl >> 32), first = 0;
                    for (int i = 0; i < n_items; i++) {
                        const int len = (blocks - first + n_items - i - 1) / (n_items - i);
                        items[at + i] = make_int4(e, b0 + first, len, 0);
                        for (int r = 0; r < len; r++) blk[b0 + first + r] = make_int2(b0 + first, len);
                        first += len;
                    }
                }
            }
            if (n_items > 0) atomicMax(&largest, (blocks + n_items - 1) / n_items * block);
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry_sh = base + incl;
        __syncthreads();
    }
    const int total = (int)(carry_sh & 0xFFFFFFFFu);
    if (thread == 0) {
        num_post[0] = total;
        if (items) {
            num_post[1] = (int)(carry_sh >> 32);
            num_post[2] = largest;
        }
    }
    for (int i = total / block + thread; i < cap / block; i += threads) expert_ids[i] = -1;
    for (int i = total + thread; i < cap; i += threads) sorted_ids[i] = numel;
    for (int i0 = 0; i0 < numel; i0 += KEEP * threads) {
        if (!one) load_ids(i0);
#pragma unroll
        for (int j = 0; j < KEEP; j++) {
            const int e = e_of[j], i = i0 + thread + j * threads;
            int at = -1;
            if (e >= 0) {
                at = offset[e] + (CL > 1 ? before[e] : 0) + (one ? rank[j] : atomicAdd(&fill[e], 1));
                sorted_ids[at] = i;
            }
            if (place && i < numel) place[i] = at;
        }
    }
}

// ------------------------------------------------------------------------------------------------ rotations

// A lane's 32 values of a row in the B-operand layout of the grouped GEMM (k chunk by k chunk of eight, a 16-byte word per row, `rows`
// rows): the warp's stores fill 128-byte lines.  The lane holds chunks q, q + 4, ...
__device__ __forceinline__ void moe_store_rows(unsigned char* unit, int rows, int row, int q, const float (&v)[32])
{
#pragma unroll
    for (int j = 0; j < 4; j++) {
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const __half2 h = __floats2half2_rn(v[8 * j + 2 * i] * HAD_SCALE, v[8 * j + 2 * i + 1] * HAD_SCALE);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(unit + ((size_t)(4 * j + q) * rows + row) * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// A lane's 32 halves of 128 (16-byte aligned) as packed words: 16-byte chunks q, q + 4, ...
__device__ __forceinline__ void moe_load32(const void* base, long long at, int q, uint32_t (&w)[16])
{
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + at) + q;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint4 r = src[4 * i];
        w[4 * i] = r.x;
        w[4 * i + 1] = r.y;
        w[4 * i + 2] = r.z;
        w[4 * i + 3] = r.w;
    }
}
// The same through shared memory, requested one column block ahead without holding registers: with 16 warps per SM (a lane's transform takes half
// of its registers) the latency of plain loads was three quarters of these kernels' time.  A warp's own: two rows per lane group, and up to three
// vectors that are the same for all its rows.  CTAs of four warps keep this within the shared memory that needs no opting in.
constexpr int MOE_HAD_WARPS = 4;
template <int ROWS>
struct MoeStage {
    uint4 row[2 * ROWS][4][32];                                          // ... and their vectors, where every row has its own (ROWS = 2)
    uint4 vec[3][16];

    static __device__ __forceinline__ void copy16(void* to, const void* from)
    {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_addr(to)), "l"(from) : "memory");
    }
    __device__ __forceinline__ void fetch_row(int r, const void* base, long long at, int lane)
    {
        const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + at) + (lane & 3);
#pragma unroll
        for (int i = 0; i < 4; i++) copy16(&row[r][i][lane], src + 4 * i);
    }
    __device__ __forceinline__ void fetch_vec(int i, const void* base, long long at, int lane)
    {
        if (lane < 16) copy16(&vec[i][lane], reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(base) + at) + lane);
    }
    static __device__ __forceinline__ void arrived()                    // what was fetched is there, for the whole warp
    {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }
    static __device__ __forceinline__ void words(const uint4* at, int step, uint32_t (&w)[16])
    {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint4 r = at[i * step];
            w[4 * i] = r.x;
            w[4 * i + 1] = r.y;
            w[4 * i + 2] = r.z;
            w[4 * i + 3] = r.w;
        }
    }
    __device__ __forceinline__ void load_row(int r, int lane, uint32_t (&w)[16]) const { words(&row[r][0][lane], 32, w); }
    __device__ __forceinline__ void load_vec(int i, int lane, uint32_t (&w)[16]) const { words(&vec[i][lane & 3], 4, w); }
};

__device__ __forceinline__ float moe_half(const uint32_t (&w)[16], int i)
{
    const __half2 h = *reinterpret_cast<const __half2*>(&w[i >> 1]);
    return i & 1 ? __high2float(h) : __low2float(h);
}

// One row per warp, four values per lane, into the same layout (fwht128's lane order).
template <int MODE>
__device__ __forceinline__ void moe_store_row(unsigned char* unit, int rows, int row, int lane, const float (&v)[4])
{
    uint32_t h[4];
#pragma unroll
    for (int e = 0; e < 4; e++) h[e] = __half_as_ushort(__float2half_rn(v[e] * HAD_SCALE));
    if constexpr (MODE == GEMV_SPLIT)
        *reinterpret_cast<uint4*>(unit + (size_t)(lane * rows + row) * 16) = make_uint4(h[0] * 0x10001u, h[1] * 0x10001u, h[2] * 0x10001u, h[3] * 0x10001u);
    else
        *reinterpret_cast<uint2*>(unit + (size_t)((lane >> 1) * rows + row) * 16 + (lane & 1) * 8) = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}
__device__ __forceinline__ void moe_load4(const void* base, long long at, bool bf16, float (&v)[4])
{
    const uint16_t* src = reinterpret_cast<const uint16_t*>(base) + at;
    uint16_t r[4];
    if ((reinterpret_cast<uintptr_t>(src) & 7) == 0) {
        const uint2 w = *reinterpret_cast<const uint2*>(src);
        r[0] = (uint16_t)w.x;
        r[1] = (uint16_t)(w.x >> 16);
        r[2] = (uint16_t)w.y;
        r[3] = (uint16_t)(w.y >> 16);
    } else {
#pragma unroll
        for (int e = 0; e < 4; e++) r[e] = src[e];
    }
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = bf16 ? __half2float(__float2half_rn(__bfloat162float(__ushort_as_bfloat16(r[e])))) : __half2float(__ushort_as_half(r[e]));
}

// Decode-sized batches, where most rows of a block of eight are padding: one warp per (row, 128 columns), as little code as possible
// (run once per launch it is bound by instruction fetch: 5 us against 7 with the form below for one token).
template <int MODE>
__global__ void __launch_bounds__(256) moe_had_in_rows_kernel(const void* __restrict__ x, int x_bf16, const __half* __restrict__ suh, int shards, int hidden,
                                                              int top_k, int numel, int cap, const int* __restrict__ sorted_ids,
                                                              const int* __restrict__ expert_ids, const int* __restrict__ num_post,
                                                              unsigned char* __restrict__ xf, long long shard_stride)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    constexpr int F_ROW = MODE == GEMV_SPLIT ? 512 : 256;
    const int lane = threadIdx.x & 31, kgs = hidden >> 7;
    const long long at = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (at >= (long long)cap * kgs) return;
    const int row = (int)(at / kgs), kg = (int)(at - (long long)row * kgs), b = row / MOE_BLOCK_ROWS;
    const int post = *num_post, slot = sorted_ids[row], ex = expert_ids[b];
    if (row >= post || slot < 0 || slot >= numel) return;
    float a[4];
    moe_load4(x, (long long)(slot / top_k) * hidden + kg * 128 + 4 * lane, x_bf16 != 0, a);
    for (int s = 0; s < shards; s++) {
        float v[4];
        moe_load4(suh, ((long long)ex * shards + s) * hidden + kg * 128 + 4 * lane, false, v);
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] *= a[e];
        fwht128(v[0], v[1], v[2], v[3], lane);
        moe_store_row<MODE>(xf + s * shard_stride + ((long long)b * kgs + kg) * MOE_BLOCK_ROWS * F_ROW, MOE_BLOCK_ROWS, row % MOE_BLOCK_ROWS, lane, v);
    }
}

template <int MODE>
__global__ void __launch_bounds__(256) moe_glu_had_in_rows_kernel(const __half* __restrict__ gu, const __half* __restrict__ suh2, int inter, int numel, int cap,
                                                                  const int* __restrict__ sorted_ids, const int* __restrict__ expert_ids,
                                                                  const int* __restrict__ num_post, unsigned char* __restrict__ xf)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    constexpr int F_ROW = MODE == GEMV_SPLIT ? 512 : 256;
    const int lane = threadIdx.x & 31, kgs = inter >> 7;
    const long long at = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (at >= (long long)cap * kgs) return;
    const int row = (int)(at / kgs), kg = (int)(at - (long long)row * kgs), b = row / MOE_BLOCK_ROWS;
    const int post = *num_post, slot = sorted_ids[row], ex = expert_ids[b];
    if (row >= post || slot < 0 || slot >= numel) return;
    const int col = kg * 128 + 4 * lane;
    float g[4], u[4], v[4];
    moe_load4(gu, (long long)slot * 2 * inter + col, false, g);
    moe_load4(gu, (long long)slot * 2 * inter + inter + col, false, u);
    moe_load4(suh2, (long long)ex * inter + col, false, v);
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] *= __half2float(__float2half_rn(g[e] / (1.0f + __expf(-g[e])) * u[e]));
    fwht128(v[0], v[1], v[2], v[3], lane);
    moe_store_row<MODE>(xf + ((long long)b * kgs + kg) * MOE_BLOCK_ROWS * F_ROW, MOE_BLOCK_ROWS, row % MOE_BLOCK_ROWS, lane, v);
}

// 32 values of a row (Had128Rows) back in the true basis: times svh, rounded to fp16 like the output of the linear.
__device__ __forceinline__ void moe_unrotate32(const Had128Rows& had, int r, const uint32_t (&sw)[16], float (&v)[32])
{
    had.row(r, v);
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __half2float(__float2half_rn(v[i] * (HAD_SCALE * moe_half(sw, i))));
}

// The kernels for long items: the transforms of 16 rows by tensor-core MMAs (Had128Rows), their inputs one column block ahead in shared memory
// (MoeStage).  A warp takes a block of eight rows (the way in: two neighbouring blocks; behind the GEMMs two column blocks, or gate and up, are
// the 16 rows) and a span of up to four column blocks, so that the chain of dependent loads (block -> expert and slot -> values) is walked once
// per span.  The span is halved while the warps are not enough for two full loads of the chip (span_of).  Bound by latency and issue together:
// 2048 tokens, 256 experts of 2048 x 512, top-8, the three kernels, thousands of cycles and millions of warp instructions, before (butterflies
// over four lanes per row, eight rows per warp, 24 warps per SM, plain loads) / with MMAs alone / one column block ahead: way in 98, 36 / 75, 21 / 71, 22; middle 61, 19 / 56, 14 /
// 48, 14; out and sum 60, 24 / 54, 17 / 49, 18.  The layer: 347 us -> 348 -> 321, 700 tokens, 64 experts of 1536 x 768, top-6 131 -> 124, 2048 tokens,
// 32 experts of 1024 x 384, top-2 67 -> 63.5.  Rows through L1 lose it again (338 us), and so does one row that all lanes without a slot ask for (700
// tokens: 137).  Padding rows are left as they are: a column of the product depends on its own row only and nothing looks at theirs.
struct MoeSpan {
    int b, kg0, kg1, slot, ex;
    bool valid, any;
    __device__ __forceinline__ MoeSpan(int span, int kgs, int cap, int numel, const int* __restrict__ sorted_ids, const int* __restrict__ expert_ids,
                                       const int* __restrict__ num_post)
    {
        const int lane = threadIdx.x & 31, spans = (kgs + span - 1) / span;
        const int at = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        b = at / spans;
        kg0 = (at - b * spans) * span;
        kg1 = kg0 + span < kgs ? kg0 + span : kgs;
        any = false;
        if (b >= cap / MOE_BLOCK_ROWS) return;
        const int post = *num_post;
        ex = expert_ids[b];
        slot = sorted_ids[b * MOE_BLOCK_ROWS + (lane >> 2)];
        any = b * MOE_BLOCK_ROWS < post;
        valid = any && slot >= 0 && slot < numel;
    }
};

// xf[shard][item][row block] = Had128(fp16(x[token(p)]) * suh[expert(p), shard]) in the B-operand layout; blockIdx.y = shard.  A warp takes two
// neighbouring blocks of eight rows, together where they are of one item and one after the other where not.
__global__ void __launch_bounds__(MOE_HAD_WARPS * 32, 4) moe_had_in_kernel(const void* __restrict__ x, int x_bf16, const __half* __restrict__ suh, int hidden, int top_k,
                                                            int numel, int cap, const int* __restrict__ sorted_ids, const int* __restrict__ expert_ids,
                                                            const int* __restrict__ num_post, const int2* __restrict__ blk,
                                                            unsigned char* __restrict__ xf, long long shard_stride, int span)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    __shared__ MoeStage<1> stages[MOE_HAD_WARPS];
    MoeStage<1>& st = stages[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, q = lane & 3, kgs = hidden >> 7, spans = (kgs + span - 1) / span;
    const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), pair = id / spans;
    const int kg0 = (id - pair * spans) * span, kg1 = kg0 + span < kgs ? kg0 + span : kgs;
    const int b0 = 2 * pair, blocks = cap / MOE_BLOCK_ROWS;
    if (b0 >= blocks) return;
    const int2 first = blk[b0];                                                   // beside the number of blocks in use, not behind it
    int2 second = blk[b0 + 1 < blocks ? b0 + 1 : b0];
    const int post = *num_post / MOE_BLOCK_ROWS;
    if (b0 >= post) return;
    if (b0 + 1 >= post) second.x = -1;
    const bool both = first.x == second.x;
#pragma unroll 1
    for (int pass = 0; pass < (both || b0 + 1 >= post ? 1 : 2); pass++) {
        const int b = b0 + pass, ex = expert_ids[b];
        const int2 run = pass ? second : first;
        const int rows = run.y * MOE_BLOCK_ROWS, row = (b - run.x) * MOE_BLOCK_ROWS + (lane >> 2);
        int slot[2];
        slot[0] = sorted_ids[b * MOE_BLOCK_ROWS + (lane >> 2)];
        slot[1] = both ? sorted_ids[(b + 1) * MOE_BLOCK_ROWS + (lane >> 2)] : -1;
        long long x_row[2];
        bool valid[2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
            valid[r] = slot[r] >= 0 && slot[r] < numel;
            x_row[r] = (long long)(valid[r] ? slot[r] / top_k : 0) * hidden;
        }
        const __half* signs = suh + ((long long)ex * gridDim.y + blockIdx.y) * hidden;
        unsigned char* unit = xf + blockIdx.y * shard_stride + ((long long)run.x * MOE_BLOCK_ROWS * kgs + (long long)kg0 * rows) * 256;
        auto fetch = [&](int kg) {
            if (valid[0]) st.fetch_row(0, x, x_row[0] + kg * 128, lane);     // not one row that every padded one would ask the same cache line for
            if (valid[1]) st.fetch_row(1, x, x_row[1] + kg * 128, lane);
            st.fetch_vec(0, signs, kg * 128, lane);
        };
        __syncwarp();
        fetch(kg0);
#pragma unroll 1
        for (int kg = kg0; kg < kg1; kg++, unit += rows * 256) {
            uint32_t xw[2][16], sw[16];
            st.arrived();
            st.load_row(0, lane, xw[0]);
            st.load_row(1, lane, xw[1]);
            st.load_vec(0, lane, sw);
            __syncwarp();
            if (kg + 1 < kg1) fetch(kg + 1);
            if (x_bf16) {
#pragma unroll
                for (int r = 0; r < 2; r++)
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const __nv_bfloat162 bb = *reinterpret_cast<const __nv_bfloat162*>(&xw[r][i]);
                        const __half2 h = __floats2half2_rn(__low2float(bb), __high2float(bb));
                        xw[r][i] = *reinterpret_cast<const uint32_t*>(&h);
                    }
            }
            Had128Rows had;
            had.run<true, true>(xw[0], xw[1], sw, lane);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                float v[32];
                had.row(r, v);
                if (valid[r]) moe_store_rows(unit, rows, row + 8 * r, q, v);
            }
        }
    }
}

// The input of the down projection: Had128( fp16( silu(gate) * up ) * suh2[expert] ) with gate | up = Had128(gu_rot[row]) * svh13[expert].
__global__ void __launch_bounds__(MOE_HAD_WARPS * 32, 4) moe_mid_kernel(const __half* __restrict__ gu_rot, const __half* __restrict__ svh13,
                                                         const __half* __restrict__ suh2, int inter, int numel, int cap,
                                                         const int* __restrict__ sorted_ids, const int* __restrict__ expert_ids,
                                                         const int* __restrict__ num_post, const int2* __restrict__ blk, unsigned char* __restrict__ xf, int span)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    __shared__ MoeStage<1> stages[MOE_HAD_WARPS];
    MoeStage<1>& st = stages[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, q = lane & 3, kgs = inter >> 7;
    const MoeSpan at(span, kgs, cap, numel, sorted_ids, expert_ids, num_post);
    if (!at.any) return;
    const int2 run = blk[at.b];
    const int rows = run.y * MOE_BLOCK_ROWS, row = (at.b - run.x) * MOE_BLOCK_ROWS + (lane >> 2);
    const __half* gu = gu_rot + (long long)run.x * MOE_BLOCK_ROWS * 2 * inter + row * 128;               // [column block][row][128]
    const __half* sv = svh13 + (long long)at.ex * 2 * inter;
    const __half* s2 = suh2 + (long long)at.ex * inter;
    unsigned char* unit = xf + ((long long)run.x * MOE_BLOCK_ROWS * kgs + (long long)at.kg0 * rows) * 256;
    auto fetch = [&](int kg) {
        st.fetch_row(0, gu, (long long)kg * rows * 128, lane);
        st.fetch_row(1, gu, (long long)(kgs + kg) * rows * 128, lane);
        st.fetch_vec(0, sv, kg * 128, lane);
        st.fetch_vec(1, sv, inter + kg * 128, lane);
        st.fetch_vec(2, s2, kg * 128, lane);
    };
    fetch(at.kg0);
#pragma unroll 1
    for (int kg = at.kg0; kg < at.kg1; kg++, unit += rows * 256) {
        uint32_t g[16], u[16], sw[16];
        st.arrived();
        st.load_row(0, lane, g);
        st.load_row(1, lane, u);
        Had128Rows had;                                       // gate and up are its two rows
        had.run<false, true>(g, u, g, lane);
        float v[32];
        st.load_vec(1, lane, sw);
        moe_unrotate32(had, 1, sw, v);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
            u[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        st.load_vec(0, lane, sw);
        moe_unrotate32(had, 0, sw, v);
        st.load_vec(2, lane, sw);
        __syncwarp();
        if (kg + 1 < at.kg1) fetch(kg + 1);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const __half2 h = __floats2half2_rn(v[2 * i] / (1.0f + __expf(-v[2 * i])) * moe_half(u, 2 * i),
                                                v[2 * i + 1] / (1.0f + __expf(-v[2 * i + 1])) * moe_half(u, 2 * i + 1));
            g[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
        had.run<true, false>(g, g, sw, lane);
        had.row(0, v);
        if (at.valid) moe_store_rows(unit, rows, row, q, v);
    }
}

// yd[slot(row), :] = fp16( Had128(yd_rot[row]) * svh2[expert] ).
__global__ void __launch_bounds__(MOE_HAD_WARPS * 32, 4) moe_out_kernel(const __half* __restrict__ yd_rot, const __half* __restrict__ svh2, int hidden, int numel, int cap,
                                                         const int* __restrict__ sorted_ids, const int* __restrict__ expert_ids,
                                                         const int* __restrict__ num_post, const int2* __restrict__ blk, __half* __restrict__ yd,
                                                         int span)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    __shared__ MoeStage<1> stages[MOE_HAD_WARPS];
    MoeStage<1>& st = stages[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, q = lane & 3;
    const MoeSpan at(span, hidden >> 7, cap, numel, sorted_ids, expert_ids, num_post);
    if (!at.any) return;
    const int2 run = blk[at.b];
    const int rows = run.y * MOE_BLOCK_ROWS, row = (at.b - run.x) * MOE_BLOCK_ROWS + (lane >> 2);
    const __half* src = yd_rot + (long long)run.x * MOE_BLOCK_ROWS * hidden + row * 128;                     // [column block][row][128]
    const __half* sv = svh2 + (long long)at.ex * hidden;
    __half* dst = yd + (long long)(at.valid ? at.slot : 0) * hidden + 8 * q;
    auto fetch = [&](int kg) {
        const int next = kg + 1 < at.kg1 ? kg + 1 : kg;
        st.fetch_row(0, src, (long long)kg * rows * 128, lane);
        st.fetch_row(1, src, (long long)next * rows * 128, lane);
    };
    fetch(at.kg0);
#pragma unroll 1
    for (int kg = at.kg0; kg < at.kg1; kg += 2) {             // two column blocks are the transform's two rows
        const bool two = kg + 1 < at.kg1;
        uint32_t w[2][16];
        st.arrived();
        st.load_row(0, lane, w[0]);
        st.load_row(1, lane, w[1]);
        __syncwarp();
        if (kg + 2 < at.kg1) fetch(kg + 2);
        Had128Rows had;
        had.run<false, true>(w[0], w[1], w[0], lane);
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (!at.valid || (r && !two)) break;
            uint32_t sw[16];
            moe_load32(sv, (kg + r) * 128, q, sw);
            float v[32];
            moe_unrotate32(had, r, sw, v);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                uint32_t o[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const __half2 h = __floats2half2_rn(v[8 * i + 2 * j], v[8 * i + 2 * j + 1]);
                    o[j] = *reinterpret_cast<const uint32_t*>(&h);
                }
                reinterpret_cast<uint4*>(dst + (kg + r) * 128)[4 * i] = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
    }
}

// y[t, :] = sum_j w[t, j] * fp16( Had128(yd_rot[place of slot t * top_k + j]) * svh2[its expert] ), in fp32, rounded to fp16 (and, for a bf16 y, from there: values
// beyond 65504 are infinite in it as well, as with explicit casts around an fp16 layer): moe_out_kernel and
// moe_combine_kernel in one, without the slots' rows in memory between.  A warp takes 8 / G tokens, G rows each (top_k rounded up to a power
// of two, at most eight; more come in rounds), four lanes per row; the rows of a token are added by exchanging halves, so that every lane ends
// with 32 / G of the 128 columns, its own.  Latency and
// issue bound it (2048 tokens, top-8, 2048 columns: 31 us under ncu for 67 MB, which are 10.4 us of traffic).  One and two rows per token spill (352 and 28
// bytes stored); top-1 gained all the same (2048 tokens, 32 experts of 2048 x 512: a layer 81 -> 74 us with the transforms on tensor cores, top-2 109 -> 99).
template <int G>
__global__ void __launch_bounds__(MOE_HAD_WARPS * 32, 4) moe_out_combine_kernel(const __half* __restrict__ yd_rot, const __half* __restrict__ svh2,
                                                                 const float* __restrict__ weights, const int* __restrict__ place,
                                                                 const int* __restrict__ expert_ids, const int2* __restrict__ blk, int tokens, int top_k,
                                                                 int hidden, void* __restrict__ y, int y_bf16, int span)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    constexpr int N = 32 / G;
    __shared__ MoeStage<2> stages[MOE_HAD_WARPS];
    MoeStage<2>& st = stages[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2, kgs = hidden >> 7, spans = (kgs + span - 1) / span;
    const int id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), group = id / spans, kg0 = (id - group * spans) * span;
    const int t = group * (8 / G) + r / G, kg1 = kg0 + span < kgs ? kg0 + span : kgs;
    if (group * (8 / G) >= tokens) return;
    const __half *src = yd_rot, *sv = svh2;
    long long pitch = 0;
    float wt = 0.f;
    bool valid = false;
    auto look = [&](int j0) {                                     // this lane's slot of a round
        const int j = j0 + r % G, slot = t * top_k + j, at = t < tokens && j < top_k ? place[slot] : -1;
        valid = at >= 0;
        if (!valid) return;
        const int b = at / MOE_BLOCK_ROWS;
        const int2 run = blk[b];
        wt = weights[slot];
        src = yd_rot + (long long)run.x * MOE_BLOCK_ROWS * hidden + (at - run.x * MOE_BLOCK_ROWS) * 128;            // [column block][row][128]
        pitch = (long long)run.y * MOE_BLOCK_ROWS * 128;
        sv = svh2 + (long long)expert_ids[b] * hidden;
    };
    look(0);
    auto fetch = [&](int kg) {
        if (!valid) return;                                       // not one row that every such lane would ask the same cache line for
        const int next = kg + 1 < kg1 ? kg + 1 : kg;
        st.fetch_row(0, src, kg * pitch, lane);
        st.fetch_row(1, src, next * pitch, lane);
        st.fetch_row(2, sv, kg * 128, lane);
        st.fetch_row(3, sv, next * 128, lane);
    };
    if (top_k <= G) fetch(kg0);
#pragma unroll 1
    for (int kg = kg0; kg < kg1; kg += 2) {                       // two column blocks are the transform's two rows
        const bool two = kg + 1 < kg1;
        float sum[2][N] = {};
#pragma unroll 1
        for (int j0 = 0; j0 < top_k; j0 += G) {
            if (top_k > G) {
                look(j0);
                fetch(kg);
            }
            uint32_t w[2][16];
            st.arrived();
            st.load_row(0, lane, w[0]);
            st.load_row(1, lane, w[1]);
            Had128Rows had;
            had.run<false, true>(w[0], w[1], w[0], lane);
#pragma unroll
            for (int b = 0; b < 2; b++) {
                if (b && !two) break;
                uint32_t sw[16];
                st.load_row(2 + b, lane, sw);
                if (top_k <= G && b == 1 && kg + 2 < kg1) fetch(kg + 2);      // what a lane fetches it alone reads
                float v[32];
                moe_unrotate32(had, b, sw, v);
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = valid ? v[i] * wt : 0.f;
#pragma unroll
                for (int m = 2 * G, n = 32; m >= 4; m >>= 1, n >>= 1) {       // lanes m apart exchange halves of n values
                    const bool upper = (lane & m) != 0;
#pragma unroll
                    for (int i = 0; i < n / 2; i++) {
                        const float keep = upper ? v[i + n / 2] : v[i], send = upper ? v[i] : v[i + n / 2];
                        v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, m);
                    }
                }
#pragma unroll
                for (int i = 0; i < N; i++) sum[b][i] += v[i];
            }
        }
#pragma unroll
        for (int b = 0; b < 2; b++) {
            if (t >= tokens || (b && !two)) break;
            uint32_t o[N / 2];
#pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const __half2 h = __floats2half2_rn(sum[b][2 * i], sum[b][2 * i + 1]);
                const __nv_bfloat162 bb = __floats2bfloat162_rn(__low2float(h), __high2float(h));
                o[i] = y_bf16 ? *reinterpret_cast<const uint32_t*>(&bb) : *reinterpret_cast<const uint32_t*>(&h);
            }
            const int at = (r % G) * N;                            // of the 32 values, whose i-th is column 32 (i / 8) + 8 q + i % 8
            uint16_t* dst = reinterpret_cast<uint16_t*>(y) + (long long)t * hidden + (kg + b) * 128 + 8 * q;
            if constexpr (N >= 8) {
#pragma unroll
                for (int i = 0; i < N / 8; i++)
                    *reinterpret_cast<uint4*>(dst + 32 * (at / 8 + i)) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            } else {
                *reinterpret_cast<uint2*>(dst + 32 * (at / 8) + at % 8) = make_uint2(o[0], o[1]);
            }
        }
    }
}

// y[t, :] = sum_j w[t, j] * yd[t*top_k + j, :] in fp32, slot order, rounded to fp16 and, for a bf16 y, from there; ids outside [0, E) are skipped.  V columns per
// thread; the rows of up to eight slots are requested together (16384 slots of 2048 columns: 40 us with two columns per thread
// and one slot at a time).
template <int V>
__global__ void __launch_bounds__(256) moe_combine_kernel(const __half* __restrict__ yd, const float* __restrict__ w, const int* __restrict__ topk_ids,
                                                          int tokens, int top_k, int hidden, int E, void* __restrict__ y, int y_bf16)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    using Vec = typename std::conditional<V == 8, uint4, uint32_t>::type;
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;       // one thread per (token, V columns)
    const int per = hidden / V;
    if (idx >= (long long)tokens * per) return;
    const int t = (int)(idx / per), c = (int)(idx - (long long)t * per) * V;
    float a[V];
#pragma unroll
    for (int i = 0; i < V; i++) a[i] = 0.f;
    for (int j0 = 0; j0 < top_k; j0 += 8) {
        Vec r[8];
        float wt[8];
        bool on[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const long long slot = (long long)t * top_k + j0 + j;
            int e = -1;
            if (j0 + j < top_k) e = topk_ids[slot];
            on[j] = e >= 0 && e < E;
            if (on[j]) {
                r[j] = *reinterpret_cast<const Vec*>(yd + slot * hidden + c);
                wt[j] = w[slot];
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (!on[j]) continue;
            const uint32_t* words = reinterpret_cast<const uint32_t*>(&r[j]);
#pragma unroll
            for (int i = 0; i < V / 2; i++) {
                const __half2 h = *reinterpret_cast<const __half2*>(&words[i]);
                a[2 * i] += wt[j] * __low2float(h);
                a[2 * i + 1] += wt[j] * __high2float(h);
            }
        }
    }
    Vec o;
    uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int i = 0; i < V / 2; i++) {
        const __half2 h = __floats2half2_rn(a[2 * i], a[2 * i + 1]);
        const __nv_bfloat162 bb = __floats2bfloat162_rn(__low2float(h), __high2float(h));
        ow[i] = y_bf16 ? *reinterpret_cast<const uint32_t*>(&bb) : *reinterpret_cast<const uint32_t*>(&h);
    }
    reinterpret_cast<Vec*>(y)[idx] = o;
}

// ------------------------------------------------------------------------------------------------ launchers

template <int K>
int launch_moe_gemm_for_k(const MoeGemmLaunch& l, int mode, int family, int grid, size_t smem, cudaStream_t st);
template <int K>
int moe_set_attributes_for_k(int max_smem);

int moe_init_device()
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    int rc = cuda_status(cudaFuncSetAttribute(moe_align_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (4 * MOE_MAX_EXPERTS + 1) * (int)sizeof(int)));
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<2>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<3>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<4>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<5>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<6>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<7>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = moe_set_attributes_for_k<8>(d->max_smem_optin);
    return rc;
}

static inline unsigned blocks_for(long long items, int per_block) { return (unsigned)((items + per_block - 1) / per_block); }

int launch_moe_align(const int* topk_ids, int numel, int E, int block, int cap, int* sorted_ids, int* expert_ids, int* num_post,
                     const int* expert_map, int E_global, int item_blocks, int4* items, int2* blk, int* header, cudaStream_t st, int* place)
{
    // Up to two slots per thread of one CTA; more are shared by a cluster (the largest portable one).
    const bool many = numel > 2048;
    return launch_chained(many ? moe_align_kernel<8> : moe_align_kernel<1>, dim3(many ? 8 : 1), dim3(1024), (size_t)((many ? 4 : 3) * E + 1) * sizeof(int), st,
                          topk_ids, numel, E, block, cap, sorted_ids, expert_ids, num_post, expert_map, E_global, item_blocks, items, blk, header, place);
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Column blocks per warp for `groups` groups of eight rows, and (span_blocks) the CTAs that this takes: up to four, as long as the warps
// fill the chip (16 per SM) twice.
static int span_of(long long groups, int cols, int least = 1)
{
    const DeviceInfo* d = current_device_info();
    const long long enough = 2 * 16 * (long long)(d ? d->sm_count : 148);
    int span = 4;
    while (span > least && groups * ((cols / 128 + span - 1) / span) < enough) span /= 2;
    return span;
}
static unsigned span_blocks(long long groups, int cols, int span) { return blocks_for(groups * ((cols / 128 + span - 1) / span), MOE_HAD_WARPS); }

int launch_moe_had_in(const void* x, int x_bf16, const __half* suh, int shards, int hidden, int top_k, int numel, int cap,
                      const int* sorted_ids, const int* expert_ids, const int* num_post, void* xf, long long shard_stride, int mode, cudaStream_t st)
{
    return launch_chained(mode == GEMV_SPLIT ? moe_had_in_rows_kernel<GEMV_SPLIT> : moe_had_in_rows_kernel<GEMV_PAIRED>,
                          dim3(blocks_for((long long)cap * (hidden / 128), 8)), dim3(256), 0, st, x, x_bf16, suh, shards, hidden, top_k, numel, cap,
                          sorted_ids, expert_ids, num_post, reinterpret_cast<unsigned char*>(xf), shard_stride);
}

int launch_moe_glu_had_in(const __half* gu, const __half* suh2, int inter, int numel, int cap, const int* sorted_ids, const int* expert_ids,
                          const int* num_post, void* xf, int mode, cudaStream_t st)
{
    return launch_chained(mode == GEMV_SPLIT ? moe_glu_had_in_rows_kernel<GEMV_SPLIT> : moe_glu_had_in_rows_kernel<GEMV_PAIRED>,
                          dim3(blocks_for((long long)cap * (inter / 128), 8)), dim3(256), 0, st, gu, suh2, inter, numel, cap, sorted_ids, expert_ids,
                          num_post, reinterpret_cast<unsigned char*>(xf));
}

int launch_moe_had_in_items(const void* x, int x_bf16, const __half* suh13, int hidden, int top_k, int numel, int cap, const int* sorted_ids,
                            const int* expert_ids, const int* num_post, const int2* blk, void* xf, long long shard_stride, cudaStream_t st)
{
    const int pairs = (cap / MOE_BLOCK_ROWS + 1) / 2, span = span_of(2 * pairs, hidden);
    return launch_chained(moe_had_in_kernel, dim3(span_blocks(pairs, hidden, span), 2), dim3(MOE_HAD_WARPS * 32), 0, st, x, x_bf16, suh13, hidden, top_k, numel, cap, sorted_ids,
                          expert_ids, num_post, blk, reinterpret_cast<unsigned char*>(xf), shard_stride, span);
}

int launch_moe_mid_items(const __half* gu_rot, const __half* svh13, const __half* suh2, int inter, int numel, int cap, const int* sorted_ids,
                         const int* expert_ids, const int* num_post, const int2* blk, void* xf, cudaStream_t st)
{
    const int groups = cap / MOE_BLOCK_ROWS, span = span_of(groups, inter);
    return launch_chained(moe_mid_kernel, dim3(span_blocks(groups, inter, span)), dim3(MOE_HAD_WARPS * 32), 0, st, gu_rot, svh13, suh2, inter, numel, cap, sorted_ids, expert_ids,
                          num_post, blk, reinterpret_cast<unsigned char*>(xf), span);
}

int launch_moe_out_items(const __half* yd_rot, const __half* svh2, int hidden, int numel, int cap, const int* sorted_ids, const int* expert_ids,
                         const int* num_post, const int2* blk, __half* yd, cudaStream_t st)
{
    const int groups = cap / MOE_BLOCK_ROWS, span = span_of(groups, hidden, 2);
    return launch_chained(moe_out_kernel, dim3(span_blocks(groups, hidden, span)), dim3(MOE_HAD_WARPS * 32), 0, st, yd_rot, svh2, hidden, numel, cap, sorted_ids, expert_ids,
                          num_post, blk, yd, span);
}

int launch_moe_out_combine(const __half* yd_rot, const __half* svh2, const float* weights, const int* place, const int* expert_ids, const int2* blk, int tokens,
                           int top_k, int hidden, void* y, int y_bf16, cudaStream_t st)
{
    const int g = top_k > 4 ? 8 : top_k > 2 ? 4 : top_k;
    auto* const kernel = g == 8 ? moe_out_combine_kernel<8> : g == 4 ? moe_out_combine_kernel<4> : g == 2 ? moe_out_combine_kernel<2> : moe_out_combine_kernel<1>;
    const int groups = (tokens + 8 / g - 1) / (8 / g), span = span_of(groups, hidden, 2);
    return launch_chained(kernel, dim3(span_blocks(groups, hidden, span)), dim3(MOE_HAD_WARPS * 32), 0, st, yd_rot, svh2, weights, place, expert_ids, blk, tokens, top_k, hidden,
                          y, y_bf16, span);
}

int launch_moe_combine(const __half* yd, const float* w, const int* topk_ids, int tokens, int top_k, int hidden, int E, void* y,
                       int y_bf16, cudaStream_t st)
{
    // Eight columns per thread once that leaves enough threads to fill the chip; few tokens are latency, not bandwidth.
    const bool wide = hidden % 8 == 0 && aligned16(yd) && aligned16(y) && (long long)tokens * hidden >= 8 * 64 * 1024;
    const int v = wide ? 8 : 2;
    return launch_chained(wide ? moe_combine_kernel<8> : moe_combine_kernel<2>, dim3(blocks_for((long long)tokens * (hidden / v), 256)), dim3(256), 0, st, yd, w,
                          topk_ids, tokens, top_k, hidden, E, y, y_bf16);
}

int launch_moe_gemm(MoeGemmLaunch l, int K, int codebook, int mode, cudaStream_t st)
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    const int grid = d->sm_count < MOE_MAX_GRID ? d->sm_count : MOE_MAX_GRID;
    // Stages of about 24 KB of weights (a bulk copy costs a few hundred nanoseconds whatever its size), a unit or more per group of decode
    // warps (see SkWalk).  Single blocks of eight rows: their activations ride with the weights, as many stages as fit; four units per stage where
    // three such stages fit, as the decode groups change stages less often (64 tokens, 256 experts: K = 4 172 -> 169 us, K = 5 191 -> 187).
    // Long items: three stages of weights, the rest for activations (larger stages take from those): of 128 rows four units and more up to K = 5, three at 6
    // and 7, two at 8.  Two stages of three units would leave them four and three there and lose all the same: 2048 tokens, 256 experts of 2048 x
    // 512, top-8, K = 6 / 7 / 8 392 / 408 / 396 us against 372 / 376 / 371; 700 tokens, 64 experts of 1536 x 768, top-6, K = 6 / 8 143.5 / 136.4 against 131 / 123
    // (half units, three stages of two: 402 / 431 / 411, 140 / 138).
    const uint32_t unit = 2048u * (uint32_t)K, row = mode == GEMV_SPLIT ? 512u : 256u, tail = MOE_BLOCK_ROWS * 128 * 4, all = (uint32_t)d->max_smem_optin;
    uint32_t ups = (24u * 1024u + unit - 1) / unit;
    if (ups < SK_GROUPS) ups = SK_GROUPS;
    uint32_t stages = 3;
    if (!l.items) {
        const uint32_t with_rows = unit + MOE_BLOCK_ROWS * row;
        if (ups < 4) ups = 4;
        while (ups > SK_GROUPS && 3 * ups * with_rows > all - MOE_BAR_BYTES - tail) ups--;
        stages = (all - MOE_BAR_BYTES - tail) / (ups * with_rows);
        if (stages > SK_MAX_STAGES) stages = SK_MAX_STAGES;
        l.x_bytes = stages * ups * MOE_BLOCK_ROWS * row;
    } else {
        l.x_bytes = (all - MOE_BAR_BYTES - tail - stages * ups * unit) & ~1023u;
    }
    l.units_per_stage = (int)ups;
    l.stages = (int)stages;
    l.x_off = MOE_BAR_BYTES + stages * ups * unit;
    l.p_off = l.x_off + l.x_bytes;
    if (l.p_off + tail > all || l.x_bytes < (uint32_t)(l.items ? MOE_TC_BLOCK_ROWS : MOE_BLOCK_ROWS) * row) return EXL3_ERR_UNSUPPORTED_ROWS;
    const CodebookConst c = codebook_const(codebook);
    l.mul = c.mul;
    l.add = c.add;
    const size_t smem = l.p_off + tail;
    const int fam = codebook_family(codebook);
    switch (K) {
        case 2: return launch_moe_gemm_for_k<2>(l, mode, fam, grid, smem, st);
        case 3: return launch_moe_gemm_for_k<3>(l, mode, fam, grid, smem, st);
        case 4: return launch_moe_gemm_for_k<4>(l, mode, fam, grid, smem, st);
        case 5: return launch_moe_gemm_for_k<5>(l, mode, fam, grid, smem, st);
        case 6: return launch_moe_gemm_for_k<6>(l, mode, fam, grid, smem, st);
        case 7: return launch_moe_gemm_for_k<7>(l, mode, fam, grid, smem, st);
        case 8: return launch_moe_gemm_for_k<8>(l, mode, fam, grid, smem, st);
    }
    return EXL3_ERR_UNSUPPORTED_K;
}

}  // namespace exl3
