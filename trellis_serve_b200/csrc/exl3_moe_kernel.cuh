// Grouped decode GEMM for routed MoE experts (sm_100a).
//
// Every (token, expert) slot is its own row because every expert has its own suh
// (cuda/src/sglang_exl3/kernels/marlin_moe.py:11-13 of 0xSero/trellis-serve).  The routing step sorts the slots by expert; an ITEM is a
// run of up to 128 rows of one expert, a multiple of eight: either the "moe blocks" of eight rows of the engine's contract
// (cuda/csrc/exl3_marlin_moe.cu:542-594), or the longer runs that launch_moe_align lists.  This kernel multiplies each item by
// its expert's matrix.  It replaces the reference's grouped Marlin instances (cuda/csrc/exl3_marlin_moe_template.h, launch at
// exl3_marlin_moe.cu:376-408), for decode batches and for prefill alike.
//
// The machinery of the dense decode GEMV (exl3_skinny_kernel.cuh): decoded registers go to tensor memory as the A operand, the rotated
// rows are the B operand (N = rows of the item), persistent CTAs split the unit list (item, column block, row block) evenly and
// contiguously, or by whole column blocks, partial sums of column blocks cut between CTAs are added in CTA order by the last one to arrive.  Two forms:
//
//   * blocks of eight rows (decode batches): the dense kernel, but for the item list that is read on the device (CUDA-graph safe), the
//     expert's svh and the scattering of rows to their slots;
//   * LIST, longer items: N and the pitch of B are run-time values, the activations have a ring of their own whose slot size follows
//     the largest item, ONE warp issues the MMAs of the three decode groups in unit order into one accumulator, so that 128 rows
//     fit into tensor memory twice; weights in paired mode only.  Rotating such rows in the epilogue would be a third of all instructions on four of 32 warps
//     (measured: 2.2 us per 32 rows, 512 x 2048 of 256 experts 192 us): they leave in the rotated basis, as fp16, and the kernels
//     behind rotate them.
//
// Bound by the issue of the decode (see exl3_skinny_kernel.cuh); the MMAs of a 16x16 tile take 8 clk at 128 paired rows.  Groups take whole units
// (three half units apart before): 256 experts of 2048 x 512, top-8, K = 3, 64 tokens 178.5 -> 175.2 us, 2048 tokens 366 -> 359.  Long items: 16.6 clk
// per tile for gate|up (16.9 before their rows left through shared memory), most of it on the scheduler that the MMA warp is on (62 instructions per tile there,
// 55 on the others): the loop that issues them frees a buffer after its own half's MMAs (not both after the unit's: 355 -> 350 us), knows
// its loop bounds as uniform (349), and is one piece of code for all groups (347).
#pragma once
#include "exl3_skinny_kernel.cuh"

namespace exl3 {

constexpr int MOE_BLOCK_ROWS = 8;
constexpr int MOE_MAX_GRID = 192;                                // CTAs of a launch (one per SM)
constexpr int MOE_ERR_WORDS = 64;                                // header of the many-row workspace: error word
constexpr int MOE_X_SLOTS = 4, MOE_X_UNITS = 4;                  // most slots of the activation ring, and units of a slot
constexpr uint32_t MOE_BAR_BYTES = 640, MOE_TABLE_OFF = 384;     // barriers, then the constants of the decode loop
// Largest expert count of one routing alignment: the form of one CTA keeps three counters per expert in the default 48 KB of shared
// memory ((3 * E + 1) * 4 bytes + 280 static), that of a cluster four in the larger size it opts in to.
constexpr int MOE_MAX_EXPERTS = 4064;

struct MoeGemmLaunch {
    const uint32_t* packed;          // [E][NB][KG][...] resident expert stack
    long long expert_stride;         // words between experts
    const unsigned char* xf;         // rotated rows: item at first row * KG * F, unit row block at + kg * rows * F, [k chunk][row] 16 bytes
    long long xf_shard_stride;       // bytes between shards
    const __half* svh;               // [E][n_total]
    __half* out;                     // fp16: [slots][n_total], or with items [item][column block][row][128] in the rotated basis
    const int* sorted_ids;           // slot of each row, >= numel for padding
    const int* expert_ids;           // expert of each block of eight rows
    const int4* items;               // (expert, first block, blocks, 0), or null: every block of eight rows is an item
    const int* counts;               // device: [0] rows; with items: [1] items, [2] rows of the largest item
    float* partials;                 // without items: [2 * grid][8][128]
    int* counters;                   // without items: [grid]
    int* err;
    int KG, NB, n_total, numel, shard_end_block;   // shard_end_block: first column block of shard 1 (NB if one shard)
    int stages, units_per_stage;
    uint32_t x_off, x_bytes, p_off;
    uint32_t mul, add;
    int rotated;                     // 1: no output Hadamard / svh (identity read-out)
};

int launch_moe_gemm(MoeGemmLaunch l, int K, int codebook, int mode, cudaStream_t st);

// Rows w and w + 4 of a block of eight (w = the epilogue warp), a row per warp at a time: from staged rows (c_last < c_first), or the
// partial sums of CTAs c_first .. c_last, added in CTA order with the loads of four CTAs in flight together.
__device__ __forceinline__ void moe_finish_eight(const MoeGemmLaunch& p, const float* src, int c_first, int c_last, uint2 sv, const int (&slots)[2], int nb,
                                                 int w, int lane)
{
    constexpr int CB = 4;
    const size_t slab = MOE_BLOCK_ROWS * 128;
    float v[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) v[i][e] = 0.f;
    const bool staged = c_last < c_first;
#pragma unroll 1
    for (int c = c_first; c <= (staged ? c_first : c_last); c += CB) {
        float4 f[CB][2];
#pragma unroll
        for (int j = 0; j < CB; j++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                f[j][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                const size_t at = (staged ? 0 : (size_t)(2 * (c + j) + (c + j == c_first)) * slab) + (w + 4 * i) * 128 + 4 * lane;
                if (staged) {
                    if (j == 0) f[j][i] = *reinterpret_cast<const float4*>(src + at);
                } else if (c + j <= c_last) {
                    f[j][i] = __ldcg(reinterpret_cast<const float4*>(src + at));
                }
            }
#pragma unroll
        for (int j = 0; j < CB; j++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                v[i][0] += f[j][i].x;
                v[i][1] += f[j][i].y;
                v[i][2] += f[j][i].z;
                v[i][3] += f[j][i].w;
            }
    }
    const __half2 s01 = *reinterpret_cast<const __half2*>(&sv.x), s23 = *reinterpret_cast<const __half2*>(&sv.y);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        if (slots[i] < 0 || slots[i] >= p.numel) continue;                  // the same for the whole warp
        if (!p.rotated) {
            fwht128(v[i][0], v[i][1], v[i][2], v[i][3], lane);
            v[i][0] *= HAD_SCALE * __low2float(s01);
            v[i][1] *= HAD_SCALE * __high2float(s01);
            v[i][2] *= HAD_SCALE * __low2float(s23);
            v[i][3] *= HAD_SCALE * __high2float(s23);
        }
        const __half2 a = __floats2half2_rn(v[i][0], v[i][1]), b = __floats2half2_rn(v[i][2], v[i][3]);
        *reinterpret_cast<uint2*>(p.out + (long long)slots[i] * p.n_total + nb * 128 + 4 * lane) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
}

// Sixteen tensor-memory lanes x sixteen columns: r[4 s .. 4 s + 3] are columns 8 s + 2 (lane % 4) and the next, of tensor-memory lane (lane / 4) and that + 8.
__device__ __forceinline__ void moe_load_turned(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// LIST: items of several blocks from the align kernel's list; otherwise every block of eight rows is an item, and row count and pitch are
// constants of the code.
template <int K, int MODE, int FAM, bool LIST>
__global__ void __launch_bounds__(SK_THREADS, 1) moe_gemm_kernel(const __grid_constant__ MoeGemmLaunch p)
{
    static_assert(!LIST || MODE == GEMV_PAIRED, "long items come with paired weights");
    constexpr int ACCS = LIST ? 1 : SK_GROUPS, NMAX = LIST ? MOE_TC_BLOCK_ROWS : 16;        // accumulators of a column block, and their columns
    constexpr uint32_t W_BYTES = 2048u * K, HALF_BYTES = K * 128u;
    constexpr uint32_t F_ROW = MODE == GEMV_SPLIT ? 512u : 256u;            // bytes of a row in a unit's activations
    constexpr int A_COLS = MODE == GEMV_SPLIT ? 64 : 32, A_OFF = 2 * ACCS * NMAX, MMAS = MODE == GEMV_SPLIT ? 8 : 4;
    static_assert(A_OFF + 2 * SK_GROUPS * A_COLS <= SK_TMEM_COLS, "tensor memory");
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* w_full = reinterpret_cast<uint64_t*>(smem);                   // weights of a stage have landed
    uint64_t* stage_empty = w_full + SK_MAX_STAGES;                         // ... have been multiplied
    uint64_t* x_full = stage_empty + SK_MAX_STAGES;                         // activations of a unit
    uint64_t* x_empty = x_full + MOE_X_SLOTS;
    uint64_t* buf_empty = x_empty + MOE_X_SLOTS;                            // [group][2] multiplied
    uint64_t* acc_done = buf_empty + 2 * SK_GROUPS;                         // LIST: [2] a column block's MMAs have completed; else [group]
    uint64_t* acc_empty = acc_done + SK_GROUPS;                             // [2] read out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* flag = reinterpret_cast<int*>(tmem_slot + 1);
    unsigned char* wring = smem + MOE_BAR_BYTES;
    unsigned char* xs = smem + p.x_off;
    float* P = reinterpret_cast<float*>(smem + p.p_off);

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int cta = blockIdx.x, ups = p.units_per_stage, stages = p.stages;
    if (warp == SK_COPY_WARP) {
        if (lane == 0) {
            for (int s = 0; s < SK_MAX_STAGES; s++) {
                ptx::mbar_init(&w_full[s], 1);
                ptx::mbar_init(&stage_empty[s], LIST ? 1 : ups);
            }
            for (int s = 0; s < MOE_X_SLOTS; s++) {
                ptx::mbar_init(&x_full[s], 1);
                ptx::mbar_init(&x_empty[s], 1);
            }
            for (int b = 0; b < 2 * SK_GROUPS; b++) ptx::mbar_init(&buf_empty[b], 1);
            for (int g = 0; g < SK_GROUPS; g++) ptx::mbar_init(&acc_done[g], 1);
            for (int d = 0; d < 2; d++) ptx::mbar_init(&acc_empty[d], 4);
            ptx::mbar_fence_init();
        }
    } else if (warp == SK_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_addr(tmem_slot)), "r"((uint32_t)SK_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x < 35)
        reinterpret_cast<uint32_t*>(smem + MOE_TABLE_OFF)[threadIdx.x] = threadIdx.x < 32 ? 1u << threadIdx.x : threadIdx.x == 32 ? p.mul : threadIdx.x == 33 ? p.add : HASH_FLIP;
    sk_fence_before();
    __syncthreads();
    sk_fence_after();
    uint32_t failed = *tmem_slot != 0;                                      // all 512 columns are this CTA's: addresses start at 0
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();                                            // the item list comes from kernels ahead in the stream

    const int UB = p.NB * p.KG;                                             // units per item
    auto uniform = [](int v) { return (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)v); };     // v >= 0, the same in every lane
    // Values read from memory go through a reduction where MMA operands depend on them: its result is a uniform register.
    const int n_items = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)(LIST ? p.counts[1] : p.counts[0] / MOE_BLOCK_ROWS));
    // What is split over the CTAs: units, or whole column blocks -- with LIST always: a row's sums are then the same whatever item the
    // alignment, whose order inside an expert is not fixed, put it into; otherwise where the exchange of partial sums that it saves is worth
    // more than what the busiest CTA takes on (the costs of the dense kernel's split, in units).
    int grain = LIST ? p.KG : 1;
    if (!LIST && (long long)n_items * UB < (1ll << 30)) {
        const unsigned blocks = (unsigned)(n_items * p.NB), cut = (blocks * p.KG + gridDim.x - 1) / gridDim.x;
        const unsigned whole = (blocks + gridDim.x - 1) / gridDim.x * p.KG;
        if (whole + (cut > 12 ? 3 : 0) < cut + 7) grain = p.KG;
    }
    const long long total = (long long)n_items * (UB / grain);
    int units_q, units_r;
    if (total < (1ll << 31)) {                                              // the 64-bit division is a few hundred clocks of everyone's start
        units_q = (int)((unsigned)total / gridDim.x);
        units_r = (int)((unsigned)total % gridDim.x);
    } else {
        units_q = (int)(total / gridDim.x);
        units_r = (int)(total % gridDim.x);
    }
    const long long u0 = gemv_first_unit(cta, units_q, units_r) * grain;
    const int units = uniform((units_q + (cta < units_r ? 1 : 0)) * grain), fills = uniform((units + ups - 1) / ups);
    // LIST, activation ring: a slot holds the activations of a run of up to x_units row blocks of a column block, consecutive in memory
    // (a bulk copy costs a few hundred nanoseconds whatever its size).
    const uint32_t x_unit = LIST ? __reduce_max_sync(0xFFFFFFFFu, (unsigned)p.counts[2]) * F_ROW : 0u;
    [[maybe_unused]] int x_units = MOE_X_UNITS, x_slots = MOE_X_SLOTS;
    if (LIST && x_unit > 0) {
        while (x_units > 1 && p.x_bytes / (x_unit * x_units) < 3) x_units--;
        x_slots = (int)(p.x_bytes / (x_unit * x_units));
        if (x_slots > MOE_X_SLOTS) x_slots = MOE_X_SLOTS;
    }
    x_units = uniform(x_units);
    x_slots = uniform(x_slots);
    [[maybe_unused]] const uint32_t slot_bytes = x_unit * x_units;
    int item = uniform(units <= 0 ? 0 : (long long)n_items * UB < (1ll << 31) ? (int)((unsigned)u0 / (unsigned)UB) : (int)(u0 / UB));
    int in_item = uniform(units > 0 ? (int)(u0 - (long long)item * UB) : 0);
    auto item_of = [&](int i) {                                             // expert, first row, rows
        if constexpr (LIST) {
            const int4 t = p.items[i];
            return make_int3(t.x, t.y * MOE_BLOCK_ROWS, t.z * MOE_BLOCK_ROWS);
        }
        else return make_int3(p.expert_ids[i], i * MOE_BLOCK_ROWS, MOE_BLOCK_ROWS);
    };

    if (warp >= SK_DECODE_WARP) {
        // ------------------------------------------------------------------ decode: as in the dense kernel, whole units
        const int dw = warp - SK_DECODE_WARP, group = dw >> 3, nt = 2 * (dw & 3) + ((dw >> 2) & 1);
        const uint32_t table = ptx::smem_addr(smem + MOE_TABLE_OFF);
        const CodebookConst cbc = {ptx::lds32(table + 128), ptx::lds32(table + 132), ptx::lds32(table + 136)};
        const int source = __shfl_sync(0xFFFFFFFFu, lane, (lane + 31) & 31);
        const SkPow2<K, FAM> pw(table);
        const uint32_t w_bar = ptx::smem_addr(w_full), ring = (uint32_t)(stages * ups) * W_BYTES;
        if (units > 0) {
            auto enter = [&](uint32_t slot8, uint32_t parity) { sk_wait(w_bar + slot8, parity, failed); };
            SkWalk at(group, ups, fills, enter);
            uint32_t wa = ptx::smem_addr(wring) + (uint32_t)(nt * 2) * HALF_BYTES + lane * 4u + group * W_BYTES;
            const uint32_t t_base = ((uint32_t)(nt * 16) << 16) + A_OFF + (uint32_t)(group * 2) * A_COLS;
            const uint32_t empty0 = ptx::smem_addr(&buf_empty[group * 2]);
            const int bar0 = SK_BAR_BUF + group * 2;
            uint32_t parity = 1;
            auto half = [&](auto which) {
                constexpr int S = decltype(which)::value;
                uint32_t L[K];
#pragma unroll
                for (int i = 0; i < K; i++) L[i] = ptx::lds32(wa + S * HALF_BYTES + i * 128u);
                constexpr int TCOLS = MODE == GEMV_SPLIT ? 16 : 8;
                const uint32_t ta = t_base + S * A_COLS;
                auto tile = [&](auto tconst) {
                    constexpr int T = decltype(tconst)::value;
                    uint32_t own[2];
                    own_words<K, T>(L, own);
                    const uint32_t prev0 = __shfl_sync(0xFFFFFFFFu, own[0], source);
                    const LaneRegs<K> R = lane_regs<K>(own, prev0);
                    uint32_t w[8];
                    decode_tile_regs<K, MODE, FAM>(R, pw, cbc, w);
                    if constexpr (MODE == GEMV_SPLIT) sk_store_tile_split(ta + T * TCOLS, w);
                    else sk_store_tile_paired(ta + T * TCOLS, w);
                };
                sk_wait(empty0 + S * 8u, parity, failed);
                sk_fence_after();
                tile(std::integral_constant<int, 0>{});
                tile(std::integral_constant<int, 1>{});
                tile(std::integral_constant<int, 2>{});
                tile(std::integral_constant<int, 3>{});
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                sk_fence_before();
                sk_bar_arrive(bar0 + S, (8 + 1) * 32);
            };
#pragma unroll 1
            for (int u = group; u < units; u += SK_GROUPS) {
                if (at.left <= 0 && at.settle(ups, stages, enter)) wa -= ring;
                half(std::integral_constant<int, 0>{});
                half(std::integral_constant<int, 1>{});
                wa += SK_GROUPS * W_BYTES;
                at.left -= SK_GROUPS;
                parity ^= 1;
            }
        }
    } else if (!LIST && warp < SK_COPY_WARP) {
        // ------------------------------------------------------------------ MMA issue, one warp per group: as in the dense kernel
        auto multiply = [&](auto gconst) {
            constexpr int group = decltype(gconst)::value;
            constexpr uint32_t F_BYTES = MOE_BLOCK_ROWS * F_ROW, chunk = MOE_BLOCK_ROWS;
            constexpr uint32_t IDESC = (1u << 4) | ((16u >> 3) << 17) | ((128u >> 4) << 24);           // fp16 x fp16 -> fp32, M = 128, N = 16
            constexpr uint32_t b_hi = (128u >> 4) | (1u << 14), a_base = A_OFF + (uint32_t)(group * 2) * A_COLS;
            const uint32_t w_bar = ptx::smem_addr(w_full), s_bar = ptx::smem_addr(stage_empty), ring = (uint32_t)(stages * ups) * F_BYTES;
            auto enter = [&](uint32_t slot8, uint32_t parity) { sk_wait(w_bar + slot8, parity, failed); };
            SkWalk at(group, ups, fills, enter);
            uint32_t xa = ptx::smem_addr(xs) + group * F_BYTES;
            const uint32_t empty0 = ptx::smem_addr(&buf_empty[group * 2]), done_bar = ptx::smem_addr(&acc_done[group]);
            uint32_t d = 0, acc_parity = 1, done_parity = 0;
            int u = group, done = 0, kg = uniform(in_item % p.KG);
#pragma unroll 1
            while (done < units) {                                          // column blocks of the CTA
                done += p.KG - kg < units - done ? p.KG - kg : units - done;
                kg = 0;
                sk_wait(ptx::smem_addr(&acc_empty[d]), acc_parity, failed);
                sk_fence_after();
                const uint32_t acc = (d * SK_GROUPS + group) * NMAX;
                uint32_t accumulate = 0;
#pragma unroll 1
                for (; u < done; u += SK_GROUPS) {
                    if (at.left <= 0 && at.settle(ups, stages, enter)) xa -= ring;
                    const uint64_t b = ((uint64_t)b_hi << 32) | (chunk << 16) | (xa >> 4);
#pragma unroll
                    for (int S = 0; S < 2; S++) {
                        ptx::named_bar_sync(SK_BAR_BUF + group * 2 + S, (8 + 1) * 32);
                        sk_fence_after();
                        if (sk_elect()) {
#pragma unroll
                            for (int m = 0; m < MMAS; m++)
                                sk_mma(acc, a_base + S * A_COLS + m * 8, b + (S * MMAS + m) * 2u * chunk, IDESC, m > 0 ? 1u : accumulate);
                            sk_commit_addr(empty0 + S * 8u);
                            if (S == 1) sk_commit_addr(s_bar + at.slot8);
                        }
                        __syncwarp();
                        accumulate = 1;
                    }
                    xa += SK_GROUPS * F_BYTES;
                    at.left -= SK_GROUPS;
                }
                if (accumulate) {                                           // else the group had no unit of this block
                    if (sk_elect()) sk_commit_addr(done_bar);
                    __syncwarp();
                    sk_wait(done_bar, done_parity, failed);
                    done_parity ^= 1;
                    sk_fence_after();
                    sk_fence_before();
                }
                sk_bar_arrive(SK_BAR_ACC + (int)d, (SK_GROUPS + 4) * 32);
                d ^= 1;
                if (d == 0) acc_parity ^= 1;
            }
        };
        if (units > 0) {
            if (warp == SK_MMA_WARP) multiply(std::integral_constant<int, 0>{});
            else if (warp == SK_MMA_WARP + 1) multiply(std::integral_constant<int, 1>{});
            else multiply(std::integral_constant<int, 2>{});
        }
    } else if (LIST && warp == SK_MMA_WARP) {
        // ------------------------------------------------------------------ MMA issue, all groups in unit order
        const uint32_t s_bar = ptx::smem_addr(stage_empty), xe_bar = ptx::smem_addr(x_empty), xf_bar = ptx::smem_addr(x_full);
        const uint32_t empty0 = ptx::smem_addr(buf_empty), done0 = ptx::smem_addr(acc_done), xs_addr = ptx::smem_addr(xs);
        uint32_t stage8 = 0, x_slot = 0, x_parity = 0, d = 0, acc_parity = 1, g = 0;
        int left = ups;
        // A unit at a time with as few instructions as possible: this warp shares its scheduler with six decode warps, whose groups wait for the
        // slowest of their members.  A half's MMAs free its buffer while the group decodes the other one.
        int done = 0;
#pragma unroll 1
        while (done < units) {                                              // column blocks of the CTA
            const int kg = uniform(in_item % p.KG), count = p.KG - kg < units - done ? p.KG - kg : units - done;
            const uint32_t pitch = __reduce_max_sync(0xFFFFFFFFu, (unsigned)item_of(item).z), chunk2 = 2u * pitch, cols = (pitch + 15u) & ~15u;
            const uint32_t idesc = (1u << 4) | ((cols >> 3) << 17) | ((128u >> 4) << 24);  // fp16 x fp16 -> fp32, M = 128, N = cols
            sk_wait(ptx::smem_addr(&acc_empty[d]), acc_parity, failed);
            sk_fence_after();
            const uint32_t acc = d * NMAX;
            uint32_t accumulate = 0;
#pragma unroll 1
            for (int todo = count; todo > 0;) {                             // runs of the activation ring
                const int run = todo < x_units ? todo : x_units;
                todo -= run;
                sk_wait(xf_bar + x_slot * 8u, x_parity, failed);
                uint32_t lo = (pitch << 16) | ((xs_addr + x_slot * slot_bytes) >> 4);
#pragma unroll 1
                for (int r = run; r > 0; r--) {
                    left--;
                    const uint32_t a = A_OFF + g * (2 * A_COLS), empty = empty0 + g * 16u;
#pragma unroll
                    for (int S = 0; S < 2; S++) {
                        ptx::named_bar_sync(SK_BAR_BUF + g * 2 + S, (8 + 1) * 32);
                        sk_fence_after();
                        if (sk_elect()) {
#pragma unroll
                            for (int m = 0; m < MMAS; m++)
                                sk_mma_at(acc, a + S * A_COLS + m * 8, lo + m * chunk2, (128u >> 4) | (1u << 14), idesc, S + m > 0 ? 1u : accumulate);
                            sk_commit_addr(empty + S * 8u);
                            if (S == 1 && r == 1) sk_commit_addr(xe_bar + x_slot * 8u);
                            if (S == 1 && left == 0) sk_commit_addr(s_bar + stage8);
                        }
                        __syncwarp();
                        lo += MMAS * chunk2;
                    }
                    accumulate = 1;
                    g = g == SK_GROUPS - 1 ? 0 : g + 1;
                    if (left == 0) {
                        left = ups;
                        stage8 = stage8 + 8 == (uint32_t)stages * 8u ? 0 : stage8 + 8;
                    }
                }
                if (++x_slot == (uint32_t)x_slots) {
                    x_slot = 0;
                    x_parity ^= 1;
                }
            }
            if (sk_elect()) sk_commit_addr(done0 + d * 8u);
            __syncwarp();
            d ^= 1;
            if (d == 0) acc_parity ^= 1;
            done += count;
            in_item += count;
            if (in_item == UB) {
                in_item = 0;
                item++;
            }
        }
    } else if (LIST && warp == SK_MMA_WARP + 1) {
        // ------------------------------------------------------------------ "column block multiplied": polls for the four epilogue warps
        uint32_t d = 0, parity = 0;
        int done = 0, kg = units > 0 ? in_item % p.KG : 0;
#pragma unroll 1
        while (done < units) {
            if (!failed && !ptx::mbar_wait_relaxed(&acc_done[d], parity, done + p.KG < units ? 400 : 60)) failed = 1;
            sk_fence_after();
            sk_fence_before();
            sk_bar_arrive(SK_BAR_ACC + (int)d, (1 + 4) * 32);
            d ^= 1;
            if (d == 0) parity ^= 1;
            done += p.KG - kg;
            kg = 0;
        }
    } else if (LIST && warp == SK_MMA_WARP + 2) {
        // ------------------------------------------------------------------ copies of activations, a run of units per slot
        if (lane == 0 && units > 0) {
            int slot = 0, runs = 0;
            uint32_t phase = 1;                                             // the first lap's slots are free
            int3 it = item_of(item);
            int nb = in_item / p.KG, kg = in_item - nb * p.KG;
            for (int j = 0; j < units; runs++) {
                int n = p.KG - kg < units - j ? p.KG - kg : units - j;
                if (n > x_units) n = x_units;
                const uint32_t unit = (uint32_t)it.z * F_ROW, bytes = (uint32_t)n * unit;
                const unsigned char* src = p.xf + (nb >= p.shard_end_block ? p.xf_shard_stride : 0) + ((long long)it.y * p.KG * F_ROW + (long long)kg * unit);
                if (!failed && !ptx::mbar_wait_relaxed(&x_empty[slot], phase, 200)) failed = 1;
                ptx::mbar_arrive_expect_tx(&x_full[slot], bytes);
                ptx::bulk_g2s(xs + (size_t)slot * slot_bytes, src, bytes, &x_full[slot]);
                if (++slot == x_slots) {
                    slot = 0;
                    phase ^= 1;
                }
                j += n;
                kg += n;
                if (kg == p.KG) {
                    kg = 0;
                    if (++nb == p.NB) {
                        nb = 0;
                        if (j < units) it = item_of(++item);
                    }
                }
            }
            for (int j = runs > x_slots ? runs - x_slots : 0; j < runs; j++) {          // every copy has landed before the CTA may leave
                uint32_t late = 0;
                sk_wait(ptx::smem_addr(&x_full[j % x_slots]), (uint32_t)(j / x_slots) & 1u, late);
                failed |= late;
            }
        }
        __syncwarp();
    } else if (warp == SK_COPY_WARP) {
        // ------------------------------------------------------------------ copies of weights; eight rows: the activations ride with them
        if (lane == 0 && units > 0) {
            int slot = 0, todo = units;
            uint32_t phase = 1;
            int e = item_of(item).x;
            [[maybe_unused]] int x_item = item, x_nb = in_item / p.KG, x_kg = in_item - x_nb * p.KG;
            for (int j = 0; j < fills; j++) {
                if (!failed && !ptx::mbar_wait_relaxed(&stage_empty[slot], phase, 400)) failed = 1;
                int n = todo < ups ? todo : ups;
                todo -= n;
                unsigned char* dst = wring + (size_t)(slot * ups) * W_BYTES;
                ptx::mbar_arrive_expect_tx(&w_full[slot], (uint32_t)n * (W_BYTES + (LIST ? 0u : MOE_BLOCK_ROWS * F_ROW)));
                [[maybe_unused]] int xn = n;
                while (n > 0) {
                    const int run = UB - in_item < n ? UB - in_item : n;     // up to the end of this expert's matrix
                    ptx::bulk_g2s(dst, p.packed + (long long)e * p.expert_stride + (long long)in_item * (512 * K), (uint32_t)run * W_BYTES, &w_full[slot]);
                    dst += (size_t)run * W_BYTES;
                    n -= run;
                    in_item += run;
                    if (in_item == UB) {
                        in_item = 0;
                        item++;
                        if (n + todo > 0) e = item_of(item).x;
                    }
                }
                if constexpr (!LIST) {
                    constexpr uint32_t F_BYTES = MOE_BLOCK_ROWS * F_ROW;
                    unsigned char* to = xs + (size_t)(slot * ups) * F_BYTES;
                    while (xn > 0) {                                        // runs of row blocks of a column block are consecutive in memory
                        const int run = p.KG - x_kg < xn ? p.KG - x_kg : xn;
                        const unsigned char* src = p.xf + (x_nb >= p.shard_end_block ? p.xf_shard_stride : 0) + ((long long)x_item * p.KG + x_kg) * F_BYTES;
                        ptx::bulk_g2s(to, src, (uint32_t)run * F_BYTES, &w_full[slot]);
                        to += (size_t)run * F_BYTES;
                        xn -= run;
                        x_kg += run;
                        if (x_kg == p.KG) {
                            x_kg = 0;
                            if (++x_nb == p.NB) {
                                x_nb = 0;
                                x_item++;
                            }
                        }
                    }
                }
                if (++slot == stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            for (int j = fills > stages ? fills - stages : 0; j < fills; j++) {
                uint32_t late = 0;
                sk_wait(ptx::smem_addr(&w_full[j % stages]), (uint32_t)(j / stages) & 1u, late);
                failed |= late;
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ epilogue
        const int ew = warp - SK_EPI_WARP, tid = (int)threadIdx.x - SK_EPI_WARP * 32;
        int d = 0, done = 0, nb = units > 0 ? in_item / p.KG : 0, kg = units > 0 ? in_item - nb * p.KG : 0;
        int3 it = make_int3(0, 0, 0);
        bool fresh = true;
#pragma unroll 1
        while (done < units) {
            const int count = p.KG - kg < units - done ? p.KG - kg : units - done;
            if (fresh) it = item_of(item);
            const bool shared = count < p.KG;                               // the column block is cut between CTAs
            int c_first = cta, c_last = cta;
            if (!LIST && shared) {
                const long long first = u0 + done - kg;                     // its first unit
                c_first = gemv_cta_of_unit(first, units_q, units_r);
                c_last = gemv_cta_of_unit(first + p.KG - 1, units_q, units_r);
            }
            [[maybe_unused]] uint2 sv = make_uint2(0u, 0u);
            [[maybe_unused]] int slots[2] = {-1, -1};
            if constexpr (!LIST) {                                          // requested while the block is still being multiplied
                if (!p.rotated) sv = *reinterpret_cast<const uint2*>(p.svh + (long long)it.x * p.n_total + nb * 128 + 4 * lane);
                slots[0] = p.sorted_ids[it.y + ew];
                slots[1] = p.sorted_ids[it.y + ew + 4];
            }
            // Tensor memory -> shared memory or the CTA's slab: lane = output column.
            const int hb = done, he = done + count;
            [[maybe_unused]] auto load_rows = [&](int c, float (&v)[8]) {
                uint32_t r[ACCS][8];
#pragma unroll
                for (int g = 0; g < ACCS; g++) sk_load8(((uint32_t)(ew * 32) << 16) + (uint32_t)((d * ACCS + g) * NMAX + c), r[g]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int g = 0; g < ACCS; g++)
#pragma unroll
                    for (int e = 0; e < 8; e++) asm volatile("" : "+r"(r[g][e]));       // no use of the registers moves ahead of the wait
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = 0.f;
#pragma unroll
                for (int g = 0; g < ACCS; g++)
                    if (hb + (g + 3 - hb % 3) % 3 < he)                     // else the group had no unit of this block
#pragma unroll
                        for (int e = 0; e < 8; e++) v[e] += __uint_as_float(r[g][e]);
            };
            [[maybe_unused]] auto read_rows = [&](int rows, float* to) {
#pragma unroll 1
                for (int c = 0; c < rows; c += 8) {
                    float v[8];
                    load_rows(c, v);
#pragma unroll
                    for (int e = 0; e < 8; e++) to[(c + e) * 128] = v[e];
                }
            };
            auto release = [&]() {
                sk_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&acc_empty[d]);
            };
            ptx::named_bar_sync(SK_BAR_ACC + d, (ACCS + 4) * 32);
            sk_fence_after();
            if (!LIST && shared) {
                constexpr size_t slab = MOE_BLOCK_ROWS * 128;
                read_rows(it.z, p.partials + (size_t)(2 * cta + (cta == c_first)) * slab + ew * 32 + lane);
                release();
                ptx::named_bar_sync(SK_BAR_EPI, 128);
                if (tid == 0) {
                    // Ordered behind every thread's partial sums by the barrier: releases them, and acquires those of the others.
                    const int last = ptx::atom_add_acq_rel_gpu(&p.counters[c_first], 1) == c_last - c_first;
                    if (last) p.counters[c_first] = 0;
                    *flag = last;
                }
                ptx::named_bar_sync(SK_BAR_EPI, 128);
                if (*flag) moe_finish_eight(p, p.partials, c_first, c_last, sv, slots, nb, ew, lane);
                ptx::named_bar_sync(SK_BAR_EPI, 128);                       // the flag may be overwritten
            } else if (!LIST) {
                read_rows(MOE_BLOCK_ROWS, P + ew * 32 + lane);
                release();
                ptx::named_bar_sync(SK_BAR_EPI, 128);
                moe_finish_eight(p, P, 0, -1, sv, slots, nb, ew, lane);
                ptx::named_bar_sync(SK_BAR_EPI, 128);
            } else {
                // Rows of a column block of an item are consecutive, [item][column block][row][128].  A warp has 32 columns of them, which come
                // out of tensor memory as pieces of rows' pairs: turned in shared memory by transposing stores of 8x8 matrices (64 bytes per
                // row, its 16-byte chunks xor-ed with the row pair: no bank conflicts) they leave as 16-byte stores.  With a column per lane and
                // two bytes per store this was 6 of 68 instructions per tile of 512 x 2048.
                const uint32_t turn = ptx::smem_addr(smem + p.p_off + ew * 1024);
                const uint32_t put = turn + (lane & 7) * 64u + (((lane >> 3) ^ (lane >> 1)) & 3) * 16u;        // row, matrix
                const uint32_t get = turn + (lane >> 2) * 64u + (((lane & 3) ^ (lane >> 3)) & 3) * 16u;        // row, chunk
                const uint32_t from = ((uint32_t)(ew * 32) << 16) + (uint32_t)(d * NMAX);
                __half* dst = p.out + (long long)it.y * p.n_total + (long long)nb * it.z * 128 + (lane >> 2) * 128 + ew * 32 + (lane & 3) * 8;
#pragma unroll 1
                for (int r0 = 0; r0 < it.z; r0 += 16) {
                    uint32_t a[2][8];                                       // columns 0 - 15 and 16 - 31 of the warp's, rows r0 .. r0 + 15
#pragma unroll
                    for (int i = 0; i < 2; i++) moe_load_turned(from + ((uint32_t)(16 * i) << 16) + r0, a[i]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 2; i++)
#pragma unroll
                        for (int e = 0; e < 8; e++) asm volatile("" : "+r"(a[i][e]));       // no use of the registers moves ahead of the wait
#pragma unroll
                    for (int s = 0; s < 2; s++) {
                        uint32_t m[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const __half2 h = __floats2half2_rn(__uint_as_float(a[j >> 1][4 * s + 2 * (j & 1)]), __uint_as_float(a[j >> 1][4 * s + 2 * (j & 1) + 1]));
                            m[j] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                        asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(put + s * 512u), "r"(m[0]), "r"(m[1]),
                                     "r"(m[2]), "r"(m[3])
                                     : "memory");
                    }
                    __syncwarp();
#pragma unroll
                    for (int s = 0; s < 2; s++)
                        if (r0 + 8 * s < it.z) {
                            uint4 v;
                            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(get + s * 512u));
                            *reinterpret_cast<uint4*>(dst + (r0 + 8 * s) * 128) = v;
                        }
                    __syncwarp();
                }
                release();
            }
            d ^= 1;
            done += count;
            kg = 0;
            fresh = ++nb == p.NB;
            if (fresh) {
                nb = 0;
                item++;
            }
        }
    }

    if (failed && lane == 0) atomicExch(p.err, GEMV_ERR_FULL_WAIT);
    sk_fence_before();
    __syncthreads();
    if (warp == SK_MMA_WARP) {
        sk_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(0u), "r"((uint32_t)SK_TMEM_COLS));
    }
}

}  // namespace exl3
