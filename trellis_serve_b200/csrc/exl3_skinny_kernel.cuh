// Decode GEMV / skinny GEMM of the EXL3 linear for 1..64 rows (sm_100a): out[r, :] = xh[r, :] @ W_inner -> optional Had128 * svh,
// W_inner decoded on the fly from the resident trellis.  The B200 counterpart of the reference's fused dense kernel
// (cuda/csrc/exl3_marlin.cu:489-527 -> cuda/csrc/exl3_marlin_template.h:271 of 0xSero/trellis-serve), built around the hardware:
//
//   * persistent grid, one CTA per SM; the (column block, row block) units of the matrix are dealt to the CTAs evenly and contiguously
//     ("stream-K"), or by column blocks or equal parts of them where that is cheaper (plan_split), so every CTA streams ONE contiguous byte
//     range of the weights, in stages of several units, with 1-D bulk async copies (TMA engine, mbarrier byte counting, no multicast)
//     issued by a copy warp;
//   * the work is the decode of the trellis, so the product must cost the decoding warps nothing: decoded registers go straight to
//     TENSOR MEMORY as the A operand of tcgen05.mma (M = 128 output columns of a column block), the rotated activations are the B
//     operand (N = rows) in shared memory.  The lane that decodes a 16x16 tile holds exactly its share of a tcgen05.st 16x256b
//     fragment: one store of eight registers per tile, no repacking.  Split mode keeps the two fp16 summands of a weight as two k
//     slots (the accumulator adds them), so every activation stands twice in a row of B; paired mode (MUL1) stores fp16 pairs;
//   * 24 decode warps in three groups of eight (one column tile each) that take whole units in turn (WHOLE; half units from three rows to
//     eight and above 16); a group decodes one half unit (64 k x 128 columns) at a time into one of its tensor-memory buffers; one MMA
//     warp per group issues the MMAs of a half unit into accumulators of its own (fixed order of additions; the epilogue adds the
//     groups' accumulators in group order).  MMAs are issued by an elected lane of
//     a CONVERGED warp with warp-uniform operands: 16 clk per MMA (N <= 32) against 47 from one thread of a diverged warp;
//   * warps that wait long wait on named barriers, which cost no issue slots: polls of mbarriers by the waiting warps were 12 of
//     67 executed instructions per tile;
//   * four epilogue warps read accumulators out, exchange the partial sums of column blocks cut between CTAs (the last CTA to arrive
//     adds them in a fixed order: deterministic, no spinning) and rotate, while the next column block is being decoded;
//   * for few rows the kernel rotates its own input -- from x, from gate | up (SiLU(gate) * up) or from the residual stream,
//     normalising it on the way -- so the linear is ONE launch.  Weights are constants: copies start, and the first half units of
//     every group are decoded, before the kernel ahead in the stream has finished.
//
// Bound by the issue of the decode and by the register ports that its pipes share: 42 to 52 instructions per 16x16 tile, whatever K (46.7 at K =
// 3, 41.7 at K = 4), are 11 to 13 clk of a SM's four schedulers; three to four more where groups take half units (49.7, 44.5).  The loop takes
// 13.8 clk per tile and SM at K = 3 (stamps in chained launches at 1.965 GHz); with half units 14.9, and 13.3 / 15.7 / 14.0 at K = 4 / 6 / 8, 16.0 and
// 16.2 for MUL1 at K = 3 and 6; 12.6 is what it takes alone, over weights that stay in shared memory and without the input rotation.  Issue
// slots are used in 64 to 72 % of a launch's active cycles.  The MMAs take 4 clk per tile of the tensor pipe at N = 16 and 8 at N = 64 and run
// beside it: 16.4 clk (K = 3) at 32 rows, 21.9 at 33 to 64, where half units are handed over in two pieces.  Chained launches over distinct
// weights, K = 3, one row, us: 5120 x 34816 41.7, 17408 x 5120 24.2, 5120 x 5120 11.0, 4096 x 4096 (K = 4) 8.5; 17408 x 5120, K = 6, MUL1, 16 rows
// 32.0.  What is not the loop, per launch at one row: 1.6 to 3.7 us from the end of the launch ahead until the input is rotated, 2.1 to 2.4 us by
// which CTAs that could not become resident early finish later than the median, 2.9 to 4.2 us from there to the stored outputs (tensor memory
// -> partial sums -> counter -> sums).  Fewer instructions in the loop's bookkeeping (one counter for stage and range, half units) changed
// nothing at K = 3 and lost 2 % at K = 4 to 8; a copy of the loop per group lost 7 % to instruction fetch.
#pragma once
#include "exl3_gemv_common.cuh"

namespace exl3 {

constexpr int SK_GROUPS = 3;
constexpr int SK_DECODE_WARPS = 8 * SK_GROUPS;
// Warp numbers.
constexpr int SK_MMA_WARP = 0;                                  // one MMA warp per group
constexpr int SK_COPY_WARP = SK_MMA_WARP + SK_GROUPS;
constexpr int SK_EPI_WARP = SK_COPY_WARP + 1;                   // four warps, aligned to four: a warp reads tensor-memory lanes 32 (warp % 4) ..
constexpr int SK_DECODE_WARP = SK_EPI_WARP + 4;                 // aligned to four as well
constexpr int SK_THREADS = (SK_DECODE_WARP + SK_DECODE_WARPS) * 32;
static_assert(SK_EPI_WARP % 4 == 0 && SK_DECODE_WARP % 4 == 0 && SK_THREADS == 1024, "roles of the skinny GEMM");
constexpr int SK_MAX_STAGES = 8;
constexpr int SK_TMEM_COLS = 512;
constexpr uint32_t SK_BAR_BYTES = 512, SK_TABLE_OFF = 320, SK_RANGE_OFF = 464, SK_DEAL_OFF = 472;
                                                                // barriers, the constants of the decode loop, a CTA's units and their deal (SK_HELD)
// Named barriers (0 is __syncthreads): the epilogue warps among themselves, "input rotated", "buffer decoded" (group x buffer),
// "column block multiplied".
constexpr int SK_BAR_EPI = 1, SK_BAR_X = 2, SK_BAR_BUF = 3, SK_BAR_ACC = 12;
constexpr int SK_FUSED_ROWS = 2;                                // largest row count with normalisation or residual stream inside
constexpr int SK_ROTATE_ROWS = 8;                               // largest row count whose input the kernel may rotate itself (16 rows measured slower)

// Where the B operand comes from: the workspace, streamed with the weights (written by a rotation or producer kernel ahead); x or
// gate | up, rotated by this kernel; the residual stream, normalised and rotated by this kernel.
enum { SK_STREAM = 0, SK_ROTATE = 1, SK_NORM = 2 };
// Which matrices: the launch's own; routed experts of every slot, or of those that have one here (see SkSlots).
enum { SK_DENSE = 0, SK_EACH = 1, SK_HELD = 2 };

// Tensor memory: accumulators [buffers][group][N columns], then the A buffers.  Every group cycles through buffers of its own: a
// wait by parity tells one fill of a barrier from the next, not from the one after, so a buffer must not pass between groups
// that may be a lap apart.  PARTS: a half unit is handed over in this many pieces (two at N = 64, where two whole ones per group do
// not fit).
template <int MODE, int N>
struct SkTmem {
    static constexpr int PARTS = MODE == GEMV_SPLIT && N > 32 ? 2 : 1;
    static constexpr int A_COLS = (MODE == GEMV_SPLIT ? 64 : 32) / PARTS;               // 32-bit columns of a buffer
    static constexpr int ACC_BUFS = N <= 16 ? 2 : 1;
    static constexpr int A_OFF = ACC_BUFS * SK_GROUPS * N;
    static constexpr int A_BUFS = 2;                                                    // per group: one filled while the other is multiplied
    static_assert(A_OFF + SK_GROUPS * A_BUFS * A_COLS <= SK_TMEM_COLS, "tensor memory");
};

// How column blocks of KG units are dealt to the CTAs.  parts == 0: pieces of `piece` units (one, or a whole column block) evenly and
// contiguously, the first units_r CTAs take units_q + 1.  parts > 0: every column block is cut into that many parts, one per CTA.
struct SkDeal {
    int grid, units_q, units_r, piece, parts;
};

// The cheapest of the three ways for `ctas` CTAs, `limit` units at most in one of them (even ranges aside); most: units of the busiest.  few: rows rotated inside in one
// pass of the decode warps.
//
// Every way of dealing the units has a cost, counted in units of the busiest CTA (0.5 us each up to 16 rows).  Partial sums that
// CTAs exchange take 2.5 us on top of whole column blocks; a range that starts and ends inside column blocks, evenly as it is, hands
// over twice: 1 us, 2 and more from nine rows up, where the hand-over is longer.  Chained launches, us, even ranges against the
// choice here: whole blocks, K = 3: 1024 x 8192 8.9 / 6.7 at one row, 1024 x 17408 10.7 / 8.6, 16.3 / 11.1 at 16, 21.2 / 17.6 at 57;
// parts: 4096 x 4096, K = 4 9.6 / 8.8, 1792 x 4096 8.7 / 6.9 at one row, 18.6 / 10.1 at 16, 27.5 / 16.0 at 57, 5120 x 5120 18.6 / 15.9
// at 16.  Where the rule stays with even ranges: 5120 x 5120, one row 11.2, in three parts (14 units for 11) 11.7; 17408 x 5120 24.9,
// 27.5; 2048 x 25088, whole blocks (32 units for 22) 18.0, 18.8.  In a long range of few rows all hand-overs but the last are hidden:
// 5120 x 34816, one row 43.3, whole blocks (80 units for 74) 44.1, but 50.0 / 46.8 at 16 rows.
__host__ __device__ inline SkDeal sk_deal(int NB, int KG, int ctas, int rows, bool few, int limit, bool aligned, int& most)
{
#ifdef __CUDA_ARCH__
    using Count = int;                                                      // of slots: far below 2^31
#else
    using Count = long long;
#endif
    const Count units = (Count)NB * KG;
    SkDeal t = {ctas, 0, 0, 1, 0};
    most = (int)((units + ctas - 1) / ctas);
    if (aligned) {
        constexpr int EXCHANGE = 5;
        const int uneven = rows > 8 ? 4 : 2, hidden = rows <= 8 && most > 12 ? 3 : 0;
        const Count whole = (Count)((NB + ctas - 1) / ctas) * KG;
        Count best = (Count)most + EXCHANGE + uneven;
        if (whole + hidden < best && whole <= limit && !(few && whole > SK_DECODE_WARPS)) {
            best = whole + hidden;
            t.piece = KG;
        }
        // Parts get shorter with their number: the fewest of the shortest that the grid has room for.  Trying each number in turn, twice per
        // call, showed in the smallest calls.
        const int room = NB < ctas ? (ctas / NB < KG ? ctas / NB : KG) : 1;
        if (room > 1) {
            const int part = (KG + room - 1) / room;
            if (part + EXCHANGE < best && part <= limit && !(few && part > SK_DECODE_WARPS)) {
                t.parts = (KG + part - 1) / part;
                t.piece = 1;
            }
        }
    }
    if (t.parts) {
        t.grid = t.parts * NB;
        most = (KG + t.parts - 1) / t.parts;
    } else {
        const Count pieces = units / t.piece;
        t.grid = pieces < ctas ? (int)pieces : ctas;
        t.units_q = (int)(pieces / t.grid);
        t.units_r = (int)(pieces % t.grid);
        most = (t.units_q + (t.units_r ? 1 : 0)) * t.piece;
    }
    return t;
}

// The units of a CTA (none for those behind a grid smaller than the one that was launched), and the CTAs that share column block nb: what the
// kernel does with the host's deal, for one that it made itself; warp-uniform to the compiler.
__device__ __forceinline__ void sk_range(const SkDeal& t, int KG, int cta, int& u0, int& u1)
{
    if (t.parts > 0) {
        const int nb = cta / t.parts, part = cta - nb * t.parts;
        u0 = nb * KG + part * KG / t.parts;
        u1 = nb * KG + (part + 1) * KG / t.parts;
    } else {
        u0 = (int)gemv_first_unit(cta, t.units_q, t.units_r) * t.piece;
        u1 = (int)gemv_first_unit(cta + 1, t.units_q, t.units_r) * t.piece;
    }
    if (cta >= t.grid) u1 = u0;
}
__device__ __forceinline__ void sk_sharers(const SkDeal& t, int KG, int cta, int nb, int& first, int& last)
{
    if (t.parts > 0) {
        first = nb * t.parts;
        last = first + t.parts - 1;
    } else if (t.piece > 1) {
        first = last = cta;
    } else {
        first = gemv_cta_of_unit((long long)nb * KG, t.units_q, t.units_r);
        last = gemv_cta_of_unit((long long)nb * KG + KG - 1, t.units_q, t.units_r);
    }
    first = __shfl_sync(0xFFFFFFFFu, first, 0);
    last = __shfl_sync(0xFFFFFFFFu, last, 0);
}

// Routed experts of a few slots as one matrix: the column blocks are runs of `blocks`, run v is the expert of slot v -- or, with a map, of the
// v-th slot that has an expert here.
struct SkSlots {
    const int* ids;             // expert of each slot (a router's)
    const int* map;             // -> this rank's or class's expert, or -1; null: as it is
    int experts, local;         // ids in [0, experts); experts behind the pointers
    int blocks, shard_blocks;   // column blocks of an expert, of one of its matrices with sign vectors of their own (gate, up)
    int per_row;                // slots that share a row of x (top-k, or 1)
    int known;                  // the ids were there before the kernel ahead began: read ahead of the wait
    long long stride;           // 32-bit words between experts

    __device__ __forceinline__ int expert(int s) const                      // without a map
    {
        const int e = __ldcg(ids + s);
        return e >= 0 && e < local ? e : -1;
    }
};

static_assert(SK_RANGE_OFF >= SK_TABLE_OFF + 35 * 4 && SK_RANGE_OFF % sizeof(int2) == 0 && SK_DEAL_OFF >= SK_RANGE_OFF + sizeof(int2) &&
                  SK_DEAL_OFF % sizeof(int) == 0 && SK_DEAL_OFF + sizeof(SkDeal) <= SK_BAR_BYTES,
              "head of the shared memory");

struct SkinnyLaunch {
    GemvArgs a;
    SkSlots s;
    int KG, NB;
    SkDeal deal;
    int stages, units_per_stage;
    uint32_t x_off, p_off;      // bytes: activations behind the weights, staged rows of the epilogue
    uint32_t r_off, r_plane;    // raw input of the in-kernel rotation (see SkRaw), bytes per plane
    long long xf_shard_stride;  // bytes between shards in xf
    unsigned long long* tl;     // measurement builds only: where this launch stamps its timeline
    uint32_t mul, add;
    int slots, most;            // slots of s; units of the busiest CTA
    uint32_t list_off;          // SK_HELD, bytes: the slots that have an expert here, (slot, expert) each
};

__device__ __forceinline__ bool sk_elect()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void sk_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void sk_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void sk_commit_addr(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// A from tensor memory, B from shared memory.
__device__ __forceinline__ void sk_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same with B's descriptor as two words.
__device__ __forceinline__ void sk_mma_at(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}\n" ::"r"(d),
        "r"(a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Rows of the operand = the tile's columns (lane / 4 and + 8), 32-bit columns = k (split) or pairs of k (paired).
__device__ __forceinline__ void sk_store_tile_split(uint32_t taddr, const uint32_t (&w)[8])
{
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[4]),
                 "r"(w[5]), "r"(w[2]), "r"(w[3]), "r"(w[6]), "r"(w[7])
                 : "memory");
}
__device__ __forceinline__ void sk_store_tile_paired(uint32_t taddr, const uint32_t (&w)[8])
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(w[0]), "r"(w[2]), "r"(w[1]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void sk_load8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// Bounded wait.  The fast path is one poll and one branch; `failed` sticks once a wait has run out (MBAR_MAX_NS), later ones then give
// up after one more poll: the control flow of every warp stays the same, the caller reports the failure at its end.
__device__ __forceinline__ void sk_wait(uint32_t bar, uint32_t parity, uint32_t& failed)
{
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u64 t, u, most;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE;\n\t"
        "mov.u64 t, %%globaltimer;\n\t"
        "setp.ne.u32 q, %0, 0;\n\t"
        "selp.u64 most, 0, %3, q;\n"
        "AGAIN:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE;\n\t"
        "mov.u64 u, %%globaltimer;\n\t"
        "sub.u64 u, u, t;\n\t"
        "setp.lt.u64 q, u, most;\n\t"
        "@q bra AGAIN;\n\t"
        "mov.u32 %0, 1;\n"
        "DONE:\n\t}"
        : "+r"(failed)
        : "r"(bar), "r"(parity), "n"(ptx::MBAR_MAX_NS)
        : "memory");
}

__device__ __forceinline__ void sk_bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// The decode loop's constants: the codebook's multiplier and addend and the powers of two of the windows of a bit rate (see
// window_low), read once per warp from shared memory.  Taken from the kernel's parameters they are fetched again for every half unit
// (7 loads of uniform registers per warp, 1.7 per tile): a shared-memory read is one that the compiler does not repeat.
template <int K, int FAM>
struct SkPow2 {
    uint32_t v[32];
    __device__ __forceinline__ SkPow2(uint32_t table)
    {
#pragma unroll
        for (int P = 0; P < 8; P++) {
            const int sh = window_at<K>(K * (7 - P)).sh;
            if (FAM == FAM_HASH && sh % 8 != 0) v[16 - sh] = ptx::lds32(table + (16 - sh) * 4);
        }
    }
};

// A group's walk over its units or half units group, group + 3, ... through the stage ring, from unit `first` on.  `left`: units left in the
// current stage, the current one included.  settle() follows it into the stage of its unit and calls enter(barrier offset, parity) for the fill.
// A ring that is used more than once has stages of three units or more (two where groups take half units), so every group has a part of
// every fill: none can be passed over, and none can be refilled before each group has seen it -- waits by parity need both.
struct SkWalk {
    int left, fills;            // units left in the stage; fills still to come
    uint32_t slot8, parity;
    template <typename F>
    __device__ __forceinline__ SkWalk(int first, int ups, int fills_, F enter) : left(ups), fills(fills_ - 1), slot8(0), parity(0)
    {
        enter(0u, 0u);
        left -= first;
    }
    // True when the walk has wrapped around to the first slot.
    template <typename F>
    __device__ __forceinline__ bool settle(int ups, int stages, F enter)
    {
        bool wrapped = false;
        while (left <= 0) {
            left += ups;
            slot8 += 8;
            if (slot8 == (uint32_t)stages * 8u) {
                slot8 = 0;
                parity ^= 1;
                wrapped = true;
            }
            if (fills-- > 0) enter(slot8, parity);
        }
        return wrapped;
    }
};

// The raw input of the CTA's units, staged in shared memory by the copy warp: planes of 256 bytes per unit -- the sign vectors, with
// SK_NORM the norm weights, then per row x (and the up half of gate | up).  Constant planes are requested before the wait for the
// kernel ahead.
struct SkRaw {
    int planes_const, planes_row;                 // planes of constants; planes per row
};
__host__ __device__ inline SkRaw sk_raw_planes(int x, int glu) { return {x == SK_NORM ? 2 : 1, glu ? 2 : 1}; }

// The decode warps turn the staged input into the B operand, one slot of RP * 512 (paired: 256) bytes per unit: one warp per unit,
// lane = four k values = one 16-byte row of a core matrix.  Rolled on purpose: code that runs once per launch is bound by instruction
// fetch.  The arithmetic is that of the rotation, activation and normalisation kernels, bit for bit.
template <int MODE, int X>
__device__ __forceinline__ void sk_rotate_input(const SkinnyLaunch& p, const unsigned char* raw, uint32_t plane, unsigned char* xs, int units,
                                                int warp, int lane)
{
    const int rows = p.a.rows;
    const bool bf16 = p.a.x_bf16 != 0, glu = X == SK_ROTATE && p.a.x_glu != 0;
    auto load4 = [&](const unsigned char* at, float (&v)[4], bool b) {
        const uint2 w = *reinterpret_cast<const uint2*>(at);
        const uint32_t r[2] = {w.x, w.y};
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const __half2 h = *reinterpret_cast<const __half2*>(&r[e]);
            const __nv_bfloat162 bb = *reinterpret_cast<const __nv_bfloat162*>(&r[e]);
            v[2 * e] = b ? __low2float(bb) : __low2float(h);
            v[2 * e + 1] = b ? __high2float(bb) : __high2float(h);
        }
    };
#pragma unroll 1
    for (int row = 0; row < rows; row++) {
        float rstd = 1.f;
        if constexpr (X == SK_NORM) rstd = gemv_row_rstd(p.a.ssq_in + (size_t)row * p.KG, p.KG, p.a.k, p.a.norm_eps, lane);
        const SkRaw planes = sk_raw_planes(X, glu);
        const unsigned char* xr = raw + (uint32_t)(planes.planes_const + row * planes.planes_row) * plane + lane * 8;
#pragma unroll 1
        for (int i = warp; i < units; i += SK_DECODE_WARPS) {
            float a[4], v[4];
            load4(xr + i * 256, a, bf16);
            if constexpr (X == SK_NORM) {
                load4(raw + plane + i * 256 + lane * 8, v, bf16);
#pragma unroll
                for (int e = 0; e < 4; e++) a[e] = gemv_round_act(a[e] * rstd * v[e], bf16);
            } else if (glu) {
                load4(xr + plane + i * 256, v, bf16);
#pragma unroll
                for (int e = 0; e < 4; e++) a[e] = gemv_round_act(a[e] / (1.0f + __expf(-a[e])) * v[e], bf16);
            }
            load4(raw + i * 256 + lane * 8, v, false);
#pragma unroll
            for (int e = 0; e < 4; e++) v[e] *= __half2float(__float2half_rn(a[e]));      // the rounding is a no-op for fp16 values
            fwht128(v[0], v[1], v[2], v[3], lane);
            uint32_t hv[4];
#pragma unroll
            for (int e = 0; e < 4; e++) hv[e] = __half_as_ushort(__float2half_rn(v[e] * HAD_SCALE));
            constexpr int RP = SK_FUSED_ROWS;
            unsigned char* slot = xs + (uint32_t)i * (RP * (MODE == GEMV_SPLIT ? 512u : 256u));
            if constexpr (MODE == GEMV_SPLIT)
                *reinterpret_cast<uint4*>(slot + (lane * RP + row) * 16) =
                    make_uint4(hv[0] * 0x10001u, hv[1] * 0x10001u, hv[2] * 0x10001u, hv[3] * 0x10001u);
            else
                *reinterpret_cast<uint2*>(slot + ((lane >> 1) * RP + row) * 16 + (lane & 1) * 8) =
                    make_uint2(hv[0] | (hv[1] << 16), hv[2] | (hv[3] << 16));
        }
    }
}

// The same for three to eight rows: a warp takes all rows of a unit, four lanes per row (fwht128_quad), so that a unit costs 64
// shuffles instead of 160 and the stores of eight rows fill whole core matrices.
template <int MODE>
__device__ __forceinline__ void sk_rotate_rows(const SkinnyLaunch& p, const unsigned char* raw, uint32_t plane, unsigned char* xs, int units,
                                               int warp, int lane)
{
    const int rows = p.a.rows;
    const bool bf16 = p.a.x_bf16 != 0;
    constexpr int RP = SK_ROTATE_ROWS;
    // Eight rows side by side in a quarter warp: its loads (planes are 16 bytes apart in the banks) are conflict-free, and so are its stores of split
    // activations; paired ones are stored eight bytes at a time, two quarter warps to the same banks.  With the four lanes of a row side by side
    // the split stores of a unit were 128 cycles of shared memory instead of 32 (5120 x 7168, five rows, K = 3 17.9 -> 17.5 us; MUL1, K = 6 18.1 -> 17.8).
    const int q = lane >> 3, row = lane & 7;
#pragma unroll 1
    for (int i = warp; i < units; i += SK_DECODE_WARPS) {
        float v[32];
        const unsigned char* signs = raw + i * 256 + q * 64;
        const unsigned char* x = raw + (uint32_t)(1 + (row < rows ? row : 0)) * plane + i * 256 + q * 64;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint4 xw = reinterpret_cast<const uint4*>(x)[j], sw = reinterpret_cast<const uint4*>(signs)[j];
            const uint32_t xv[4] = {xw.x, xw.y, xw.z, xw.w}, sv[4] = {sw.x, sw.y, sw.z, sw.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                __half2 h = *reinterpret_cast<const __half2*>(&xv[e]);
                if (bf16) {
                    const __nv_bfloat162 bb = *reinterpret_cast<const __nv_bfloat162*>(&xv[e]);
                    h = __floats2half2_rn(__low2float(bb), __high2float(bb));
                }
                const __half2 s = *reinterpret_cast<const __half2*>(&sv[e]);
                v[8 * j + 2 * e] = __low2float(s) * __low2float(h);
                v[8 * j + 2 * e + 1] = __high2float(s) * __high2float(h);
            }
        }
        fwht128_quad<8>(v, lane);
        if (row < rows) {
            unsigned char* slot = xs + (uint32_t)i * (RP * (MODE == GEMV_SPLIT ? 512u : 256u)) + row * 16;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                uint32_t hv[4];
#pragma unroll
                for (int e = 0; e < 4; e++) hv[e] = __half_as_ushort(__float2half_rn(v[4 * j + e] * HAD_SCALE));
                if constexpr (MODE == GEMV_SPLIT)
                    *reinterpret_cast<uint4*>(slot + (q * 8 + j) * (RP * 16)) =
                        make_uint4(hv[0] * 0x10001u, hv[1] * 0x10001u, hv[2] * 0x10001u, hv[3] * 0x10001u);
                else
                    *reinterpret_cast<uint2*>(slot + (q * 4 + (j >> 1)) * (RP * 16) + (j & 1) * 8) = make_uint2(hv[0] | (hv[1] << 16), hv[2] | (hv[3] << 16));
            }
        }
    }
}

// The finished sums of column block nb -> output, rows w, w + nw, ... of a warp.  shared: the block's partial sums of CTAs c_first ..
// c_last are added in CTA order; several rows and CTAs are requested together, so that their round trips overlap.
// svh: so that svh + 128 nb_out are the block's; nb_out: where it stands in the output.
template <int RB, int EPI>
__device__ __forceinline__ void sk_finish_block(const GemvArgs& a, const __half* svh, uint32_t tp_epoch, const float* P, bool shared, int c_first, int c_last,
                                                int nb, int nb_out, int w, int nw, int lane)
{
    constexpr int CB = 8 / RB;
    const int rows = a.rows;
    const size_t nelem = (size_t)rows * 128;
    const int last = shared ? c_last : 0;
#pragma unroll 1
    for (int m = w; m < rows; m += nw * RB) {
        float v[RB][4];
        const float* src = (shared ? a.partials + (size_t)(c_first + nb) * nelem : P) + m * 128 + 4 * lane;
#pragma unroll
        for (int i = 0; i < RB; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) v[i][e] = 0.f;
#pragma unroll 1
        for (int c = shared ? c_first : 0; c <= last; c += CB, src += CB * nelem) {
            float4 f[CB][RB];
#pragma unroll
            for (int j = 0; j < CB; j++)
#pragma unroll
                for (int i = 0; i < RB; i++) {
                    f[j][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (m + nw * i < rows && (j == 0 || c + j <= last)) {
                        const float4* at = reinterpret_cast<const float4*>(src + j * nelem + (size_t)(nw * i) * 128);
                        f[j][i] = shared ? __ldcg(at) : *at;
                    }
                }
#pragma unroll
            for (int j = 0; j < CB; j++)
#pragma unroll
                for (int i = 0; i < RB; i++) {
                    v[i][0] += f[j][i].x;
                    v[i][1] += f[j][i].y;
                    v[i][2] += f[j][i].z;
                    v[i][3] += f[j][i].w;
                }
        }
#pragma unroll 1
        for (int i = 0; i < RB; i++) {
            if (m + nw * i < rows) gemv_finish_row<EPI>(a, svh, tp_epoch, make_float4(v[0][0], v[0][1], v[0][2], v[0][3]), m + nw * i, nb_out, lane);
#pragma unroll
            for (int j = 0; j + 1 < RB; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) v[j][e] = v[j + 1][e];
        }
    }
}

template <int RB, int EPI>
static __device__ __noinline__ void sk_finish_block_call(const GemvArgs& a, uint32_t tp_epoch, const float* P, bool shared, int c_first, int c_last,
                                                         int nb, int w, int nw, int lane)
{
    sk_finish_block<RB, EPI>(a, a.svh, tp_epoch, P, shared, c_first, c_last, nb, nb, w, nw, lane);
}

// RP: operand pitch, the rows rounded up (operand_pitch).
// WHOLE: a group takes whole units, not every third half unit: one walk through the stages, one loop test and addresses that are constants for eight
// tiles instead of four (49.7 -> 46.7 instructions per tile at K = 3, the loop 14.9 -> 13.8 clk).  Chained launches over distinct weights, K = 3, one
// row, us: 5120 x 34816 42.7 -> 41.7, 17408 x 5120 24.7 -> 24.2, 2048 x 25088 17.3 -> 17.0, 4096 x 4096 8.8 -> 8.6; 17408 x 5120 at K = 2, 4, 5, 6, 7, 8
// 24.5 -> 23.9, 23.6 -> 23.2, 26.0 -> 25.7, 25.9 -> 25.3, 26.7 -> 26.4, 25.4 -> 25.1, MUL1 26.4 -> 25.5; 16 rows 30.6 -> 30.1, MUL1 at K = 6 33.0 ->
// 32.0.  What it costs: at the end of a column block a group may be a unit behind the others
// instead of half of one, which shows where a CTA has few units in two blocks (5120 x 7168, 15 units: one row 13.65 -> 13.75, but five rows 17.7 ->
// 18.4, as its sums of the first block then hold up the second).  Hence not for three to eight rows, most of whose launches, those that rotate inside, have such
// ranges; longer ones of that many rows, whose activations are streamed, were not tried.  Above 16 rows a stage of three units takes too
// much shared memory.
// SLOTS: the matrix is that of SkSlots, one row per slot, rotated inside.  SK_EACH: every slot as it stands; one whose id is out of range decodes
// expert 0 and drops the result.  SK_HELD, for ids with a map (a rank's share of the experts, bitrate classes): every CTA makes the same list of
// the slots that have an expert here, and where that is not all of them their units are dealt anew, so that the others cost nothing: 256
// experts of 2048 x 512, top-8, K = 3, us per layer in a chain, a rank with 128 / 64 / 32 of them: one token 21.8 / 16.7 / 13.6, two tokens
// 25.4 / 21.2 / 16.0 (every slot decoded 23.3 / 23.0 / 22.5 and 31.4 / 31.2 / 30.7, blocks of eight rows 29.9 / 23.5 / 19.3 and 32.5 / 29.5 /
// 24.1); four classes of 64, two tokens 70 (108).  Where every slot has an expert the list costs 0.3 us a layer (20.8, 21.1 with it), which is
// why SK_EACH stays.
template <int K, int MODE, int FAM, int RP, int X = SK_STREAM, int EPI = 0, int SLOTS = SK_DENSE>
__global__ void __launch_bounds__(SK_THREADS, 1) skinny_kernel(const __grid_constant__ SkinnyLaunch p)
{
    static_assert((X != SK_NORM && EPI == 0) || RP == SK_FUSED_ROWS, "the kernel normalises, and carries the residual stream of, one or two rows");
    static_assert(SLOTS == SK_DENSE || (X == SK_ROTATE && RP == SK_FUSED_ROWS && EPI == 0), "slots come one row each");
    static_assert(X != SK_ROTATE || RP <= SK_ROTATE_ROWS, "the kernel rotates up to eight rows");
    constexpr int RB = RP <= 8 ? 1 : RP <= 16 ? 2 : 4;                      // rows that a warp finishes together
    constexpr bool ALL_FINISH = RP >= 16, WHOLE = RP != SK_ROTATE_ROWS && RP <= 16;
    constexpr int N = RP < 16 ? 16 : RP;                                    // MMA columns; those behind the real rows are never looked at
    using TM = SkTmem<MODE, N>;
    constexpr uint32_t W_BYTES = 2048u * K, HALF_BYTES = K * 128u;
    constexpr uint32_t F_BYTES = (uint32_t)RP * (MODE == GEMV_SPLIT ? 512u : 256u);        // a unit's activations
    constexpr int MMAS = (MODE == GEMV_SPLIT ? 8 : 4) / TM::PARTS;          // per buffer
    constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);      // fp16 x fp16 -> fp32, M = 128
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* w_full = reinterpret_cast<uint64_t*>(smem);                   // weights of a stage have landed
    uint64_t* x_full = w_full + SK_MAX_STAGES;                              // ... its activations (rotation inside: [0] raw input, [1] constants)
    uint64_t* stage_empty = x_full + SK_MAX_STAGES;                         // its half units have been multiplied
    uint64_t* buf_empty = stage_empty + SK_MAX_STAGES;                      // [group][A_BUFS] multiplied
    uint64_t* acc_done = buf_empty + TM::A_BUFS * SK_GROUPS;                // [group] a column block's MMAs have completed
    uint64_t* acc_empty = acc_done + SK_GROUPS;                             // [ACC_BUFS] read out
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* flag = reinterpret_cast<int*>(tmem_slot + 1);
    unsigned char* wring = smem + SK_BAR_BYTES;
    unsigned char* xs = smem + p.x_off;
    float* P = reinterpret_cast<float*>(smem + p.p_off);                    // [rows][128]

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp-uniform to the compiler
    const int cta = blockIdx.x, rows = p.a.rows;
    int u0, u1;                                                             // units [u0, u1)
    if (p.deal.parts > 0) {
        const int nb = cta / p.deal.parts, part = cta - nb * p.deal.parts;
        u0 = nb * p.KG + part * p.KG / p.deal.parts;
        u1 = nb * p.KG + (part + 1) * p.KG / p.deal.parts;
    } else {
        u0 = (int)gemv_first_unit(cta, p.deal.units_q, p.deal.units_r) * p.deal.piece;
        u1 = (int)gemv_first_unit(cta + 1, p.deal.units_q, p.deal.units_r) * p.deal.piece;
    }
    // SK_HELD: the slots that have an expert here, and what the copy warp made of them.
    [[maybe_unused]] int2* list = reinterpret_cast<int2*>(smem + p.list_off);
    [[maybe_unused]] SkDeal* dealt = reinterpret_cast<SkDeal*>(smem + SK_DEAL_OFF);
    [[maybe_unused]] int2* range = reinterpret_cast<int2*>(smem + SK_RANGE_OFF);
    [[maybe_unused]] auto run_of = [&](int v) { return SLOTS == SK_HELD ? list[v] : make_int2(v, p.s.expert(v)); };      // (slot, expert or -1)
    auto sharers = [&](int nb, int& first, int& last) {                     // CTAs that share column block nb
        if constexpr (SLOTS == SK_HELD) {
            sk_sharers(*dealt, p.KG, cta, nb, first, last);
        } else if (p.deal.parts > 0) {
            first = nb * p.deal.parts;
            last = first + p.deal.parts - 1;
        } else if (p.deal.piece > 1) {
            first = last = cta;
        } else {
            first = gemv_cta_of_unit((long long)nb * p.KG, p.deal.units_q, p.deal.units_r);
            last = gemv_cta_of_unit((long long)nb * p.KG + p.KG - 1, p.deal.units_q, p.deal.units_r);
        }
    };
    const int ups = p.units_per_stage, stages = p.stages;
    int units = u1 - u0, halves = 2 * units, fills = (u1 - u0 + ups - 1) / ups;

    auto weights = [&](int j, int slot) {                                   // one thread: fill number j, units [u0 + j * ups, ...)
        const int u = u0 + j * ups, n = u1 - u < ups ? u1 - u : ups;
        ptx::mbar_arrive_expect_tx(&w_full[slot], (uint32_t)n * W_BYTES);
        if constexpr (SLOTS != SK_DENSE) {
            const int per = p.s.blocks * p.KG;                              // units of an expert
            unsigned char* dst = wring + (size_t)(slot * ups) * W_BYTES;
            for (int at = u; at < u + n;) {
                const int sl = at / per, in = at - sl * per, run = per - in < u + n - at ? per - in : u + n - at, e = run_of(sl).y;
                ptx::bulk_g2s(dst, p.a.packed + (e < 0 ? 0 : e) * p.s.stride + (long long)in * (512 * K), (uint32_t)run * W_BYTES, &w_full[slot]);
                dst += (size_t)run * W_BYTES;
                at += run;
            }
        } else {
            ptx::bulk_g2s(wring + (size_t)(slot * ups) * W_BYTES, p.a.packed + (long long)u * (512 * K), (uint32_t)n * W_BYTES, &w_full[slot]);
        }
    };
    // One thread: the CTA's units' 256 bytes of sign vectors, or (row >= 0) of plane `row` of the input, of the slots' experts.
    [[maybe_unused]] auto rows_of_slots = [&](unsigned char* dst, int row, uint64_t* bar) {
        for (int u = u0; u < u1;) {
            const int unb = u / p.KG, ukg = u - unb * p.KG, run = p.KG - ukg < u1 - u ? p.KG - ukg : u1 - u;
            const int v = unb / p.s.blocks, nb = unb - v * p.s.blocks;
            const unsigned char* src;
            if (row >= 0) {
                const int slot = SLOTS == SK_HELD ? list[v].x : v;
                src = reinterpret_cast<const unsigned char*>(p.a.x) + ((long long)(slot / p.s.per_row) * sk_raw_planes(X, p.a.x_glu).planes_row + row) * 2 * p.a.k;
            } else {
                const int e = run_of(v).y;
                src = reinterpret_cast<const unsigned char*>(p.a.suh) + ((long long)(e < 0 ? 0 : e) * (p.s.blocks / p.s.shard_blocks) + nb / p.s.shard_blocks) * 2 * p.a.k;
            }
            ptx::bulk_g2s(dst, src + ukg * 256, (uint32_t)run * 256u, bar);
            dst += (size_t)run * 256;
            u += run;
        }
    };
    // One thread: n units from u on, `bytes` per row block of a column block (consecutive in memory), a source per shard.
    auto rows_of = [&](int u, int n, unsigned char* dst, const void* src, uint32_t bytes, long long shard_stride, uint64_t* bar) {
        while (n > 0) {
            const int unb = u / p.KG, ukg = u - unb * p.KG;
            int run = p.KG - ukg, s = 0;
            if (run > n) run = n;
            while (s < p.a.n_shards - 1 && unb >= p.a.shard_end_blocks[s]) s++;
            ptx::bulk_g2s(dst, reinterpret_cast<const unsigned char*>(src) + s * shard_stride + (long long)ukg * bytes, (uint32_t)run * bytes, bar);
            dst += (size_t)run * bytes;
            u += run;
            n -= run;
        }
    };
    EXL3_STAMP(0);
    if (warp == SK_COPY_WARP) {
        auto constants = [&]() {                                            // one thread: before the kernel ahead has finished
            for (int j = 0; j < stages && j < fills; j++) weights(j, j);
            if constexpr (X != SK_STREAM) {
                const int n = u1 - u0;
                ptx::mbar_arrive_expect_tx(&x_full[1], (uint32_t)(n * sk_raw_planes(X, 0).planes_const) * 256u);
                if constexpr (SLOTS != SK_DENSE) rows_of_slots(smem + p.r_off, -1, &x_full[1]);
                else rows_of(u0, n, smem + p.r_off, p.a.suh, 256, 2ll * p.a.k, &x_full[1]);
                if constexpr (X == SK_NORM) rows_of(u0, n, smem + p.r_off + p.r_plane, p.a.norm_weight, 256, 0, &x_full[1]);
            }
        };
        if (lane == 0) {
            for (int s = 0; s < SK_MAX_STAGES; s++) {
                ptx::mbar_init(&w_full[s], 1);
                ptx::mbar_init(&x_full[s], 1);
                ptx::mbar_init(&stage_empty[s], WHOLE ? ups : 2 * ups);
            }
            for (int b = 0; b < TM::A_BUFS * SK_GROUPS; b++) ptx::mbar_init(&buf_empty[b], 1);
            for (int g = 0; g < SK_GROUPS; g++) ptx::mbar_init(&acc_done[g], 1);
            for (int d = 0; d < TM::ACC_BUFS; d++) ptx::mbar_init(&acc_empty[d], 4);
            ptx::mbar_fence_init();
            if constexpr (SLOTS == SK_EACH) {
                if (!p.s.known) ptx::grid_dependency_wait();                // the ids
            }
            if constexpr (SLOTS != SK_HELD) constants();
        }
        if constexpr (SLOTS == SK_HELD) {
            SkDeal t = p.deal;
            int held = 0;
            auto look = [&](int s0, auto count) {                           // 32 `count` slots whose round trips overlap
                constexpr int C = decltype(count)::value;
                int e[C];
#pragma unroll
                for (int i = 0; i < C; i++) e[i] = s0 + 32 * i + lane < p.slots ? __ldcg(p.s.ids + s0 + 32 * i + lane) : -1;
#pragma unroll
                for (int i = 0; i < C; i++) e[i] = e[i] >= 0 && e[i] < p.s.experts ? __ldcg(p.s.map + e[i]) : -1;
#pragma unroll
                for (int i = 0; i < C; i++) {
                    const bool has = e[i] >= 0 && e[i] < p.s.local;
                    const uint32_t have = __ballot_sync(0xFFFFFFFFu, has);
                    if (has) list[held + __popc(have & ((1u << lane) - 1))] = make_int2(s0 + 32 * i + lane, e[i]);
                    held += __popc(have);
                }
            };
            if (!p.s.known) ptx::grid_dependency_wait();                    // the ids
            if (p.slots <= 32) {
                look(0, std::integral_constant<int, 1>{});
            } else {
#pragma unroll 1
                for (int s0 = 0; s0 < p.slots; s0 += 128) look(s0, std::integral_constant<int, 4>{});
            }
            if (held < p.slots) {
                int most;
                t = {0, 0, 0, 1, 0};
                if (held > 0) t = sk_deal(held * p.s.blocks, p.KG, (int)gridDim.x, 1, false, p.most, true, most);
                sk_range(t, p.KG, cta, u0, u1);
                fills = (u1 - u0 + ups - 1) / ups;
            }
            __syncwarp();
            if (lane == 0) {
                if (u0 < u1) constants();
                *dealt = t;
                *range = make_int2(u0, u1);
            }
        }
    } else if (warp == SK_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_addr(tmem_slot)), "r"((uint32_t)SK_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x < 35)
        reinterpret_cast<uint32_t*>(smem + SK_TABLE_OFF)[threadIdx.x] = threadIdx.x < 32 ? 1u << threadIdx.x : threadIdx.x == 32 ? p.mul : threadIdx.x == 33 ? p.add : HASH_FLIP;
    sk_fence_before();
    __syncthreads();
    sk_fence_after();
    // All 512 columns are this CTA's: tensor memory starts at address 0, which keeps the addresses warp-uniform constants.
    uint32_t failed = *tmem_slot != 0;
    if constexpr (SLOTS == SK_HELD) {
        // Warp-uniform to the compiler, as the host's deal is: the loops of the MMA warps run over these (1.3 us a layer otherwise).
        const int2 mine = *range;
        u0 = __shfl_sync(0xFFFFFFFFu, mine.x, 0);
        u1 = __shfl_sync(0xFFFFFFFFu, mine.y, 0);
        units = u1 - u0;
        halves = 2 * units;
        fills = (u1 - u0 + ups - 1) / ups;
    }
    if constexpr (SLOTS != SK_DENSE) {
        // The kernel behind may look at the ids as soon as it begins: not before the kernel that wrote them has finished.
        if (!p.s.known) ptx::grid_dependency_wait();
    }
    ptx::grid_launch_dependents();                                          // the next kernel in the stream may begin its prologue

    if (SLOTS == SK_HELD && u0 >= u1) {
        ptx::grid_dependency_wait();                                        // nothing for this CTA
    } else if (warp >= SK_DECODE_WARP) {
        // ------------------------------------------------------------------ decode
        const int dw = warp - SK_DECODE_WARP, group = dw >> 3, nt = 2 * (dw & 3) + ((dw >> 2) & 1);  // columns 16 nt .. = tensor-memory lanes of this warp's quarter
        const uint32_t table = ptx::smem_addr(smem + SK_TABLE_OFF);
        const CodebookConst cbc = {ptx::lds32(table + 128), ptx::lds32(table + 132), ptx::lds32(table + 136)};
        const int source = __shfl_sync(0xFFFFFFFFu, lane, (lane + 31) & 31);      // from a shuffle, or the addition is made again per tile
        const SkPow2<K, FAM> pw(table);
        const uint32_t w_bar = ptx::smem_addr(w_full), ring = (uint32_t)(stages * ups) * W_BYTES;
        auto enter = [&](uint32_t slot8, uint32_t parity) { sk_wait(w_bar + slot8, parity, failed); };
        SkWalk at(WHOLE ? group : group >> 1, ups, fills, enter);
        uint32_t wa = ptx::smem_addr(wring) + (uint32_t)(nt * 2) * HALF_BYTES + lane * 4u +
                      (WHOLE ? group * W_BYTES : (group >> 1) * W_BYTES + (group & 1) * HALF_BYTES);
        const uint32_t t_base = ((uint32_t)(nt * 16) << 16) + TM::A_OFF + (uint32_t)(group * TM::A_BUFS) * TM::A_COLS;
        const uint32_t empty0 = ptx::smem_addr(&buf_empty[group * TM::A_BUFS]);
        const int bar0 = SK_BAR_BUF + group * TM::A_BUFS;
        uint32_t parity = 1;
        int h = group;
        // Every step moves by three halves: a group's halves alternate between the two of a unit, and between its two buffers.
        const uint32_t move0 = group & 1 ? 2 * W_BYTES - HALF_BYTES : W_BYTES + HALF_BYTES, move1 = 3 * W_BYTES - move0;
        const int adv0 = 1 + (group & 1);
        auto step = [&](auto which) {
            constexpr int S = decltype(which)::value;
            // A stage is waited for when its first unit is wanted, not before: stages behind the first lap come only once units have been
            // multiplied, and with the rotation inside that takes every decode warp.
            if ((!WHOLE || S == 0) && at.left <= 0 && at.settle(ups, stages, enter)) wa -= ring;
            uint32_t L[K];
#pragma unroll
            for (int i = 0; i < K; i++) L[i] = ptx::lds32(wa + (WHOLE ? S * HALF_BYTES : 0u) + i * 128u);
            auto tile = [&](auto tconst, uint32_t ta) {
                constexpr int T = decltype(tconst)::value;
                uint32_t own[2];
                own_words<K, T>(L, own);
                const uint32_t prev0 = __shfl_sync(0xFFFFFFFFu, own[0], source);
                const LaneRegs<K> R = lane_regs<K>(own, prev0);
                uint32_t w[8];
                decode_tile_regs<K, MODE, FAM>(R, pw, cbc, w);
                if constexpr (MODE == GEMV_SPLIT) sk_store_tile_split(ta, w);
                else sk_store_tile_paired(ta, w);
            };
            constexpr int TCOLS = MODE == GEMV_SPLIT ? 16 : 8;              // columns of a tile
            constexpr int B0 = TM::PARTS == 1 ? S : 0;                      // buffer of the first (or only) piece
            auto open = [&](int buf, uint32_t par) {
                sk_wait(empty0 + buf * 8u, par, failed);
                sk_fence_after();
            };
            auto close = [&](int buf) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                sk_fence_before();
                sk_bar_arrive(bar0 + buf, (8 + 1) * 32);
            };
            open(B0, parity);
            tile(std::integral_constant<int, 0>{}, t_base + B0 * TM::A_COLS);
            tile(std::integral_constant<int, 1>{}, t_base + B0 * TM::A_COLS + TCOLS);
            if constexpr (TM::PARTS == 1) {
                tile(std::integral_constant<int, 2>{}, t_base + B0 * TM::A_COLS + 2 * TCOLS);
                tile(std::integral_constant<int, 3>{}, t_base + B0 * TM::A_COLS + 3 * TCOLS);
                close(B0);
            } else {
                close(0);
                open(1, parity);
                tile(std::integral_constant<int, 2>{}, t_base + TM::A_COLS);
                tile(std::integral_constant<int, 3>{}, t_base + TM::A_COLS + TCOLS);
                close(1);
                if (S == 0) parity ^= 1;
            }
            if constexpr (!WHOLE) {
                wa += S == 0 ? move0 : move1;
                at.left -= S == 0 ? adv0 : 3 - adv0;
                h += SK_GROUPS;
            } else if constexpr (S == 1) {
                wa += SK_GROUPS * W_BYTES;
                at.left -= SK_GROUPS;
                h += SK_GROUPS;
            }
        };
        const int n = WHOLE ? units : halves;
        EXL3_STAMP_LANE(dw == 0, 3);
        [[maybe_unused]] bool rotated = false;
#pragma unroll 1
        while (true) {
            if (h < n) {
                step(std::integral_constant<int, 0>{});
                if (WHOLE || h < n) step(std::integral_constant<int, 1>{});
                parity ^= 1;
            }
            if constexpr (X != SK_STREAM) {
                if (!rotated) {                                             // both buffers are full, or there is nothing more to decode
                    ptx::grid_dependency_wait();
                    EXL3_STAMP_LANE(dw == 0, 1);
                    sk_wait(ptx::smem_addr(&x_full[1]), 0, failed);
                    sk_wait(ptx::smem_addr(&x_full[0]), 0, failed);
                    if constexpr (RP > SK_FUSED_ROWS) sk_rotate_rows<MODE>(p, smem + p.r_off, p.r_plane, xs, u1 - u0, dw, lane);
                    else sk_rotate_input<MODE, X>(p, smem + p.r_off, p.r_plane, xs, u1 - u0, dw, lane);
                    EXL3_STAMP_LANE(dw == 0, 2);
                    fence_async_shared();                                   // -> visible to the tensor core's reads
                    sk_bar_arrive(SK_BAR_X, (SK_DECODE_WARPS + SK_GROUPS) * 32);
                    rotated = true;
                }
            }
            if (h >= n) break;
        }
        EXL3_STAMP_LANE(dw == 0, 4);
        ptx::grid_dependency_wait();
    } else if (warp < SK_COPY_WARP) {
        // ------------------------------------------------------------------ MMA issue, one warp per group
        ptx::grid_dependency_wait();
        if constexpr (X != SK_STREAM) ptx::named_bar_sync(SK_BAR_X, (SK_DECODE_WARPS + SK_GROUPS) * 32);
        else EXL3_STAMP_LANE(warp == SK_MMA_WARP, 1);
        // The group is a constant of each warp's code, so that every operand of the MMAs is warp-uniform to the compiler.
        auto multiply = [&](auto gconst) {
            constexpr int group = decltype(gconst)::value;
            const uint32_t x_bar = ptx::smem_addr(x_full), s_bar = ptx::smem_addr(stage_empty), ring = (uint32_t)(stages * ups) * F_BYTES;
            auto enter = [&](uint32_t slot8, uint32_t parity) {
                if constexpr (X == SK_STREAM) sk_wait(x_bar + slot8, parity, failed);
            };
            SkWalk at(WHOLE ? group : group >> 1, ups, fills, enter);
            if constexpr (X == SK_STREAM && group == 0) EXL3_STAMP_LANE(true, 2);
            uint32_t xa = ptx::smem_addr(xs) + (WHOLE ? group * F_BYTES : (group >> 1) * F_BYTES + (group & 1) * (F_BYTES / 2));
            constexpr uint32_t chunk = RP;                                  // 16-byte rows between chunks of 8 k slots
            constexpr uint32_t b_hi = (128u >> 4) | (1u << 14);             // 8-row groups 128 bytes apart; descriptor version
            constexpr uint32_t a_base = TM::A_OFF + (uint32_t)(group * TM::A_BUFS) * TM::A_COLS;
            const uint32_t empty0 = ptx::smem_addr(&buf_empty[group * TM::A_BUFS]), done = ptx::smem_addr(&acc_done[group]);
            uint32_t d = 0, acc_parity = 1, done_parity = 0;
            int h = group;
            uint32_t acc = 0, accumulate = 0;
            auto step = [&](auto which) {                                   // the steps of the decode warps (see there)
                constexpr int S = decltype(which)::value;
                constexpr uint32_t half = S == 0 ? group & 1 : 1 - (group & 1);
                constexpr int PIECES = WHOLE ? 2 : TM::PARTS;
                if (at.left <= 0 && at.settle(ups, stages, enter) && X == SK_STREAM) xa -= ring;
                uint64_t b = ((uint64_t)b_hi << 32) | (chunk << 16) | (xa >> 4);
#pragma unroll
                for (int part = 0; part < PIECES; part++) {
                    constexpr int B0 = PIECES == 1 ? S : 0;
                    const int buf = B0 + part;
                    ptx::named_bar_sync(SK_BAR_BUF + group * TM::A_BUFS + buf, (8 + 1) * 32);
                    sk_fence_after();
                    if (sk_elect()) {
#pragma unroll
                        for (int m = 0; m < MMAS; m++)
                            sk_mma(acc, a_base + buf * TM::A_COLS + m * 8, b + m * 2u * chunk, IDESC, m > 0 ? 1u : accumulate);
                        sk_commit_addr(empty0 + buf * 8u);
                        if (part == PIECES - 1) sk_commit_addr(s_bar + at.slot8);
                    }
                    __syncwarp();
                    accumulate = 1;
                    b += MMAS * 2u * chunk;
                }
                xa += WHOLE ? SK_GROUPS * F_BYTES : half ? 2 * F_BYTES - F_BYTES / 2 : F_BYTES + F_BYTES / 2;
                at.left -= WHOLE ? SK_GROUPS : 1 + half;
                h += SK_GROUPS;
            };
            [[maybe_unused]] bool second = false;                                            // which of the two steps comes next
#pragma unroll 1
            for (int ub = u0; ub < u1;) {                                   // column blocks of the CTA
                const int left = p.KG - ub % p.KG, ue = ub + left < u1 ? ub + left : u1, he = (WHOLE ? 1 : 2) * (ue - u0);
                sk_wait(ptx::smem_addr(&acc_empty[d]), acc_parity, failed);
                sk_fence_after();
                acc = (d * SK_GROUPS + group) * N;
                accumulate = 0;
#pragma unroll 1
                while (h < he) {
                    if constexpr (WHOLE) {
                        step(std::integral_constant<int, 0>{});
                        continue;
                    }
                    if (!second) {
                        step(std::integral_constant<int, 0>{});
                        if (h >= he) {
                            second = true;
                            break;
                        }
                    }
                    step(std::integral_constant<int, 1>{});
                    second = false;
                }
                if (accumulate) {                                           // else the group had no half unit of this block
                    if (sk_elect()) sk_commit_addr(done);
                    __syncwarp();
                    sk_wait(done, done_parity, failed);
                    done_parity ^= 1;
                    sk_fence_after();
                    sk_fence_before();
                }
                sk_bar_arrive(SK_BAR_ACC + (int)d, (SK_GROUPS + 4) * 32);
                if (++d == TM::ACC_BUFS) {
                    d = 0;
                    acc_parity ^= 1;
                }
                ub = ue;
            }
        };
        if (warp == SK_MMA_WARP) multiply(std::integral_constant<int, 0>{});
        else if (warp == SK_MMA_WARP + 1) multiply(std::integral_constant<int, 1>{});
        else multiply(std::integral_constant<int, 2>{});
    } else if (warp == SK_COPY_WARP) {
        // ------------------------------------------------------------------ copies
        if (lane == 0) {
            auto activations = [&](int j, int slot) {                       // fill number j of the streamed activations
                const int u = u0 + j * ups, n = u1 - u < ups ? u1 - u : ups;
                ptx::mbar_arrive_expect_tx(&x_full[slot], (uint32_t)n * F_BYTES);
                rows_of(u, n, xs + (size_t)(slot * ups) * F_BYTES, p.a.xf, F_BYTES, p.xf_shard_stride, &x_full[slot]);
            };
            ptx::grid_dependency_wait();
            if constexpr (X == SK_STREAM) {
                for (int j = 0; j < stages && j < fills; j++) activations(j, j);
            } else {
                const int n = u1 - u0, row_planes = sk_raw_planes(X, p.a.x_glu).planes_row;
                const unsigned char* x = reinterpret_cast<const unsigned char*>(p.a.x);
                unsigned char* dst = smem + p.r_off + sk_raw_planes(X, p.a.x_glu).planes_const * p.r_plane;
                ptx::mbar_arrive_expect_tx(&x_full[0], (uint32_t)(n * rows * row_planes) * 256u);
                for (int q = 0; q < rows * row_planes; q++, x += 2 * p.a.k, dst += p.r_plane) {
                    if constexpr (SLOTS != SK_DENSE) rows_of_slots(dst, q, &x_full[0]);
                    else rows_of(u0, n, dst, x, 256, 0, &x_full[0]);
                }
            }
            int slot = 0;
            uint32_t phase = 0;
            for (int j = stages; j < fills; j++) {
                if (!failed && !ptx::mbar_wait_relaxed(&stage_empty[slot], phase, 100)) failed = 1;      // stages ahead of the decode: in no hurry
                weights(j, slot);
                if constexpr (X == SK_STREAM) activations(j, slot);
                if (++slot == stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            // Every copy has landed before the CTA may leave, also when a wait elsewhere has given up.
            for (int j = fills > stages ? fills - stages : 0; j < fills; j++) {
                const uint32_t lap = (uint32_t)(j / stages) & 1u;
                uint32_t late = 0;
                sk_wait(ptx::smem_addr(&w_full[j % stages]), lap, late);
                if constexpr (X == SK_STREAM) sk_wait(ptx::smem_addr(&x_full[j % stages]), lap, late);
                failed |= late;
            }
            if constexpr (X != SK_STREAM) {
                sk_wait(ptx::smem_addr(&x_full[1]), 0, failed);
                sk_wait(ptx::smem_addr(&x_full[0]), 0, failed);
            }
        }
        __syncwarp();
        ptx::grid_dependency_wait();
    } else {
        // ------------------------------------------------------------------ epilogue
        ptx::grid_dependency_wait();
        const int ew = warp - SK_EPI_WARP, tid = (int)threadIdx.x - SK_EPI_WARP * 32;
        const uint32_t tp_epoch = p.a.tp.world > 1 ? (uint32_t)*reinterpret_cast<volatile int*>(p.a.tp.state) + 1u : 0u;
        int d = 0;
        for (int ub = u0; ub < u1;) {
            const int nb = ub / p.KG, left = (nb + 1) * p.KG - ub, ue = ub + left < u1 ? ub + left : u1;
            const int hb = (WHOLE ? 1 : 2) * (ub - u0), he = (WHOLE ? 1 : 2) * (ue - u0);     // units, or half units
            int c_first, c_last;
            sharers(nb, c_first, c_last);
            const bool shared = c_first != c_last;
            const size_t nelem = (size_t)rows * 128;
            float* dst = (shared ? p.a.partials + (size_t)(cta + nb) * nelem : P) + ew * 32 + lane;
            const __half* svh = p.a.svh;
            int nb_out = nb;
            [[maybe_unused]] bool held = true;                              // SLOTS: the slot has an expert
            if constexpr (SLOTS != SK_DENSE) {
                const int v = nb / p.s.blocks;
                const int2 run = run_of(v);
                held = run.y >= 0;
                nb_out += (run.x - v) * p.s.blocks;
                svh += (long long)(run.y - run.x) * p.s.blocks * 128;
            }
            ptx::named_bar_sync(SK_BAR_ACC + d, (SK_GROUPS + 4) * 32);
            sk_fence_after();
#pragma unroll 1
            for (int c = 0; c < N && c < rows; c += 8) {
                uint32_t r[SK_GROUPS][8];
#pragma unroll
                for (int g = 0; g < SK_GROUPS; g++) sk_load8(((uint32_t)(ew * 32) << 16) + (uint32_t)((d * SK_GROUPS + g) * N + c), r[g]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int g = 0; g < SK_GROUPS; g++)
#pragma unroll
                    for (int e = 0; e < 8; e++) asm volatile("" : "+r"(r[g][e]));       // no use of the registers moves ahead of the wait
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = 0.f;
#pragma unroll
                for (int g = 0; g < SK_GROUPS; g++)
                    if (hb + (g + 3 - hb % 3) % 3 < he)                     // else the group had no half unit of this block
#pragma unroll
                        for (int e = 0; e < 8; e++) v[e] += __uint_as_float(r[g][e]);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    if (c + e < rows) dst[(c + e) * 128] = v[e];
            }
            sk_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&acc_empty[d]);
            if (++d == TM::ACC_BUFS) d = 0;
            ptx::named_bar_sync(SK_BAR_EPI, 128);
            bool finish = true;
            if (shared) {
                if (tid == 0) {
                    // The barrier ordered every thread's partial sums before this update, which releases them (and, for the last CTA to
                    // arrive, acquires those of the others ahead of the barrier below): one round trip, no separate fences.
                    const int last = ptx::atom_add_acq_rel_gpu(&p.a.counters[nb], 1) == c_last - c_first;
                    if (last) p.a.counters[nb] = 0;          // leave the counter ready for the next launch
                    *flag = last;
                }
                ptx::named_bar_sync(SK_BAR_EPI, 128);
                EXL3_STAMP_LANE(ew == 0, 6);
                finish = *flag != 0;
            }
            // From nine rows up the last block of the CTA is finished by all warps (below), which have nothing else to do by then.
            if (ALL_FINISH && ue == u1) {
                if (tid == 0) *flag = finish;
                break;
            }
            if (finish && held) {
                if constexpr (ALL_FINISH) sk_finish_block_call<RB, EPI>(p.a, tp_epoch, P, shared, c_first, c_last, nb, ew, 4, lane);
                else sk_finish_block<RB, EPI>(p.a, svh, tp_epoch, P, shared, c_first, c_last, nb, nb_out, ew, 4, lane);
            }
            EXL3_STAMP_LANE(ew == 0, 7);
            ptx::named_bar_sync(SK_BAR_EPI, 128);                           // staged rows and flag may be overwritten
            ub = ue;
        }
    }

    if (failed && lane == 0) atomicExch(p.a.err, GEMV_ERR_FULL_WAIT);
    sk_fence_before();
    __syncthreads();
    if (warp == SK_MMA_WARP) {
        sk_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(0u), "r"((uint32_t)SK_TMEM_COLS) : "memory");
    }
    const uint32_t tp_epoch = p.a.tp.world > 1 ? (uint32_t)*reinterpret_cast<volatile int*>(p.a.tp.state) + 1u : 0u;
    if (ALL_FINISH && *flag) {
        const int nb = (u1 - 1) / p.KG;
        int c_first, c_last;
        sharers(nb, c_first, c_last);
        sk_finish_block_call<RB, EPI>(p.a, tp_epoch, P, c_first != c_last, c_first, c_last, nb, warp, SK_THREADS / 32, lane);
    }
    EXL3_STAMP(5);
    if (p.a.tp.world > 1) {
        // The call number moves on once every CTA of this launch has read it: the last CTA to get here bumps it.
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&p.a.tp.state[2], 1) == (int)gridDim.x - 1) {
                p.a.tp.state[2] = 0;
                p.a.tp.state[0] = (int)tp_epoch;
            }
        }
    }
}

template <int K>
int launch_skinny_for_k(const SkinnyLaunch& l, int pitch, int x, size_t smem, cudaStream_t st);
template <int K>
int skinny_set_attributes_for_k(int max_smem);

}  // namespace exl3
