// EXL3 trellis decode primitives for sm_100a: lane-local window extraction for any K in 2..8, the three
// computed codebooks, and a 128-point Walsh-Hadamard transform held in one warp.
//
// Written from the format description, not from the reference's kernels.  What each piece corresponds to in
// 0xSero/trellis-serve:
//   windows / bit order   core/src/trellis_core/reference.py:81-99   (cuda/csrc/exl3_decode.cuh:149-360 for K=3..6)
//   codebooks             core/src/trellis_core/reference.py:53-73   (cuda/csrc/third_party/exllamav3/codebook.cuh:56-123)
//   tile placement        core/src/trellis_core/reference.py:30-45
//   Hadamard              core/src/trellis_core/reference.py:119-130 (cuda/csrc/exl3_had.cuh:20-84)
//
// Resident ("packed") layout used by every kernel here.  It is a pure permutation of the stored bits, so
// the packed-weight byte count is unchanged (k*n*K/8):
//
//   packed[nb][kg][nt][kq][i][lane]   uint32
//     nb   = output column block of 128            (n / 128)
//     kg   = input row block of 128                (k / 128)
//     nt   = 16-column tile inside the block       (8)
//     kq   = group of four 16-row tiles            (2)
//     i    = word of the lane's stream             (K)
//     lane = 32
//
// The "lane stream" of (nb, kg, nt, kq, lane) is B0|B1|B2|B3, where Bt are stream bits [8K*lane, 8K*(lane+1))
// of tile (row tile kg*8 + kq*4 + t, column tile nb*8 + nt), first stream bit in the most significant
// position.  Lane `lane` therefore owns stream elements 8*lane .. 8*lane+7 of each of its four tiles; the
// 16-K bits that element 8*lane also needs from the previous lane arrive by one warp shuffle per tile.
// One (nb, kg) unit is 2048*K contiguous bytes: a bulk-copy friendly stage.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

namespace exl3 {

constexpr int CB_3INST = 0;
constexpr int CB_MCG = 1;
constexpr int CB_MUL1 = 2;

constexpr uint32_t MUL_3INST = 89226354u;
constexpr uint32_t ADD_3INST = 64248484u;
constexpr uint32_t MUL_MCG = 0xCBAC1FEDu;
constexpr uint32_t MUL_MUL1 = 0x83DCD12Du;

// Codebook family as the kernels see it: the two "hash" codebooks differ only in two constants.
constexpr int FAM_HASH = 0;   // 3INST, MCG: x = s*mul + add; (x & 0x8FFF8FFF) ^ 0x3B603B60; value = lo + hi
constexpr int FAM_MUL1 = 1;   // MUL1: x = s*mul; value = fma(half(0x6400 + bytesum(x)), 0x1EEE, 0xC931)

constexpr uint32_t HASH_MASK = 0x8FFF8FFFu, HASH_FLIP = 0x3B603B60u;

struct CodebookConst {
    uint32_t mul;
    uint32_t add;
    uint32_t flip = HASH_FLIP;
};

__host__ __device__ inline CodebookConst codebook_const(int cb)
{
    if (cb == CB_3INST) return {MUL_3INST, ADD_3INST};
    if (cb == CB_MCG) return {MUL_MCG, 0u};
    return {MUL_MUL1, 0u};
}

__host__ __device__ inline int codebook_family(int cb) { return cb == CB_MUL1 ? FAM_MUL1 : FAM_HASH; }

// ---------------------------------------------------------------------------------------------- bit helpers

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// 32 bits of the lane stream L (K words, bit b of the stream = bit 31-(b%32) of word b/32) that end at bit
// position END (exclusive), right-aligned.  Bits before the start of the stream read as zero.
template <int K, int END>
__device__ __forceinline__ uint32_t stream_bits_ending_at(const uint32_t (&L)[K])
{
    static_assert(END > 0 && END <= 32 * K, "window end outside the lane stream");
    constexpr int wi = END / 32;
    constexpr int r = END % 32;
    if constexpr (r == 0) {
        return L[wi - 1];
    } else if constexpr (wi == 0) {
        return L[0] >> (32 - r);
    } else {
        return __funnelshift_l(L[wi], L[wi - 1], r);
    }
}

// The lane's view of one tile: E = (last 16-K bits of the previous lane's share) | (own 8K bits),
// right-aligned in up to three words.  Element p (0..7) of the lane is E bits [K*(7-p), K*(7-p)+16).
template <int K>
struct LaneTile {
    uint32_t e[3];
};

// Own share of tile T (0..3) right-aligned: word 0 = last 32 own bits, word 1 = the 32 before, ...
// Words above the own share contain neighbouring bits of the stream; assemble() masks or replaces them.
template <int K, int T>
__device__ __forceinline__ void own_words(const uint32_t (&L)[K], uint32_t (&o)[2])
{
    constexpr int END = 8 * K * (T + 1);
    o[0] = stream_bits_ending_at<K, END>(L);
    if constexpr (8 * K > 32) {
        o[1] = stream_bits_ending_at<K, END - 32>(L);
    } else {
        o[1] = 0;
    }
}

// own: this lane's right-aligned words; prev0: word 0 of the previous lane's right-aligned share of the same tile.
template <int K>
__device__ __forceinline__ LaneTile<K> assemble(const uint32_t (&own)[2], uint32_t prev0)
{
    LaneTile<K> t;
    if constexpr (K == 2) {            // own 16 bits
        t.e[0] = prmt(own[0], prev0, 0x5410);
        t.e[1] = 0;
        t.e[2] = 0;
    } else if constexpr (K == 3) {     // own 24 bits
        t.e[0] = prmt(own[0], prev0, 0x4210);
        t.e[1] = prev0 >> 8;
        t.e[2] = 0;
    } else if constexpr (K == 4) {     // own 32 bits
        t.e[0] = own[0];
        t.e[1] = prev0;
        t.e[2] = 0;
    } else if constexpr (K == 5) {     // own 40 bits
        t.e[0] = own[0];
        t.e[1] = prmt(own[1], prev0, 0x6540);
        t.e[2] = 0;
    } else if constexpr (K == 6) {     // own 48 bits
        t.e[0] = own[0];
        t.e[1] = prmt(own[1], prev0, 0x5410);
        t.e[2] = 0;
    } else if constexpr (K == 7) {     // own 56 bits
        t.e[0] = own[0];
        t.e[1] = prmt(own[1], prev0, 0x4210);
        t.e[2] = prev0 >> 8;
    } else {                           // K == 8, own 64 bits
        t.e[0] = own[0];
        t.e[1] = own[1];
        t.e[2] = prev0;
    }
    return t;
}

// 16-bit trellis state of element P (0..7) of the lane.
template <int K, int P>
__device__ __forceinline__ uint32_t window(const LaneTile<K>& t)
{
    constexpr int lo = K * (7 - P);
    constexpr int wi = lo / 32;
    constexpr int sh = lo % 32;
    if constexpr (sh == 0) {
        return t.e[wi] & 0xFFFFu;
    } else if constexpr (sh == 16) {
        return t.e[wi] >> 16;
    } else if constexpr (sh + 16 <= 32) {
        return (t.e[wi] >> sh) & 0xFFFFu;
    } else {
        return __funnelshift_r(t.e[wi], t.e[wi + 1], sh) & 0xFFFFu;
    }
}

// ---------------------------------------------------------------------------------------------- windows in few instructions
//
// The decode loops are bound by instruction issue, so a window is cut out of 32-bit registers of E that are chosen per bit rate:
//
//   * a window at bit 0, 8 or 16 of a register costs one instruction (mask, byte permute, shift);
//   * any other costs two: one multiply by a power of two (drops the bits above the window, FMA pipe) and one shift right by 16 (drops
//     those below, ALU pipe) -- shift and mask would put both on the ALU pipe, the busier of the two;
//   * a register costs one instruction (permute or funnel shift) unless the lane's words are it already.
//
// Registers and windows together: 12 / 16 / 11 / 16 / 16 / 16 / 10 instructions per tile and lane at K = 2 .. 8, against 15 / 17 / 13 / 17 /
// 16 / 19 / 10 with registers at E[16 j, 16 j + 32) (17408 x 5120, one row, chained launches: K = 5 27.2 -> 25.8 us, K = 7 29.4 -> 27.0, K =
// 3, 4 and 6 1 to 2 % less, K = 2 and 8 the same).  The powers of two come from kernel parameters (constant bank) or from shared memory
// so that the multiply stays a multiply.

struct Pow2 {
    uint32_t v[32];          // v[c] = 1 << c
};

__host__ inline Pow2 make_pow2()
{
    Pow2 p;
    for (int c = 0; c < 32; c++) p.v[c] = 1u << c;
    return p;
}

// Register and bit offset at which the window of E bits [lo, lo + 16) is found.
struct WindowAt {
    int reg, sh;
};

template <int K>
__host__ __device__ constexpr WindowAt window_at(int lo)
{
    if (K == 2) return {(lo & 7) >> 1, lo & 8};
    if (K == 3) return lo < 8 ? WindowAt{0, lo} : WindowAt{1, lo - 8};
    if (K == 4) return lo == 12 || lo >= 20 ? WindowAt{1, lo - 12} : WindowAt{0, lo};
    if (K == 5) return lo < 20 ? WindowAt{0, lo} : WindowAt{1, lo - 20};
    if (K == 6) return lo < 18 ? WindowAt{0, lo} : lo < 36 ? WindowAt{1, lo - 18} : WindowAt{2, lo - 32};
    if (K == 7) return lo < 21 ? WindowAt{0, lo} : lo < 42 ? WindowAt{1, lo - 21} : WindowAt{2, lo - 40};
    return lo <= 16 ? WindowAt{0, lo} : lo == 24 ? WindowAt{1, 8} : lo <= 48 ? WindowAt{2, lo - 32} : WindowAt{3, 8};
}

template <int K>
struct LaneRegs {
    uint32_t r[4];           // see window_at
};

// own: this lane's right-aligned words; prev0: word 0 of the previous lane's right-aligned share of the same tile.
template <int K>
__device__ __forceinline__ LaneRegs<K> lane_regs(const uint32_t (&own)[2], uint32_t prev0)
{
    LaneRegs<K> R;
    R.r[0] = own[0];
    R.r[1] = R.r[2] = R.r[3] = 0;
    if constexpr (K == 2) {                                  // own 16 bits
        R.r[0] = prmt(own[0], prev0, 0x5410);
        R.r[1] = R.r[0] >> 2;
        R.r[2] = R.r[0] >> 4;
        R.r[3] = R.r[0] >> 6;
    } else if constexpr (K == 3) {                           // own 24
        R.r[1] = prmt(own[0], prev0, 0x5421);                // E[8, 40)
    } else if constexpr (K == 4) {                           // own 32
        R.r[1] = __funnelshift_r(own[0], prev0, 12);
    } else if constexpr (K == 5) {                           // own 40
        R.r[1] = __funnelshift_r(own[0], prmt(own[1], prev0, 0x6540), 20);
    } else if constexpr (K == 6) {                           // own 48
        R.r[1] = __funnelshift_r(own[0], own[1], 18);
        R.r[2] = prmt(own[1], prev0, 0x5410);                // E[32, 64)
    } else if constexpr (K == 7) {                           // own 56
        R.r[1] = __funnelshift_r(own[0], own[1], 21);
        R.r[2] = prmt(own[1], prev0, 0x5421);                // E[40, 72)
    } else {                                                 // own 64
        R.r[1] = prmt(own[0], own[1], 0x5432);               // E[16, 48)
        R.r[2] = own[1];
        R.r[3] = prmt(own[1], prev0, 0x5432);                // E[48, 80)
    }
    return R;
}

// 16-bit trellis state of element P (0..7) of the lane, bits above it cleared.  MUL1 spends two multiplies and half an fp16 multiply-add
// per weight on the FMA pipe already, so its windows are cut with shift and mask (17408 x 5120, one row, K = 3 / 6: 28.6 -> 26.4 and
// 29.6 -> 28.0 us); for the hash codebooks the same costs 2 us.
template <int K, int P, int FAM, typename Powers>
__device__ __forceinline__ uint32_t window_low(const LaneRegs<K>& R, const Powers& pw)
{
    constexpr WindowAt at = window_at<K>(K * (7 - P));
    static_assert(at.sh >= 0 && at.sh <= 16, "window outside its register");
    if constexpr (at.sh == 0) return R.r[at.reg] & 0xFFFFu;
    else if constexpr (at.sh == 8) return prmt(R.r[at.reg], 0u, 0x4421);
    else if constexpr (at.sh == 16) return R.r[at.reg] >> 16;
    else if constexpr (FAM == FAM_MUL1) return (R.r[at.reg] >> at.sh) & 0xFFFFu;
    else return (R.r[at.reg] * pw.v[16 - at.sh]) >> 16;
}

// ---------------------------------------------------------------------------------------------- codebooks

// Hash codebooks: the register holds two fp16 numbers whose sum is the weight.
__device__ __forceinline__ uint32_t hash_pair(uint32_t state, CodebookConst c)
{
    // One multiply-add and ONE three-input logic op, (a & mask) ^ flip, with the mask as its immediate: a logic op of three registers
    // beside a multiply-add of three takes register ports that the two pipes share (register-only loop of multiply, shift, multiply-add
    // and logic op: 100 lanes/clk/SM against 108; with a multiplier from the constant bank 112).
    uint32_t x = state * c.mul + c.add, d;
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(d) : "r"(x), "n"(HASH_MASK), "r"(c.flip));
    return d;
}

// One weight, fp16, rounded once: bit-identical to the codebook table of the reference decoder.
__device__ __forceinline__ __half decode_value(uint32_t state, int family, CodebookConst c)
{
    if (family == FAM_HASH) {
        uint32_t x = hash_pair(state, c);
        __half2 h = *reinterpret_cast<__half2*>(&x);
        return __hadd(__low2half(h), __high2half(h));
    }
    uint32_t x = state * c.mul;
    uint32_t bits = __dp4a(x, 0x01010101u, 0x6400u);
    __half h = __ushort_as_half(static_cast<unsigned short>(bits));
    return __hfma(h, __ushort_as_half(0x1EEE), __ushort_as_half(0xC931));
}

// Two MUL1 weights at once: states a, b -> half2(value(a), value(b)).
__device__ __forceinline__ uint32_t mul1_pair(uint32_t sa, uint32_t sb, CodebookConst c)
{
    uint32_t ha = __dp4a(sa * c.mul, 0x01010101u, 0x6400u);
    uint32_t hb = __dp4a(sb * c.mul, 0x01010101u, 0x6400u);
    uint32_t packed = prmt(ha, hb, 0x5410);
    __half2 h = *reinterpret_cast<__half2*>(&packed);
    const __half2 m = __half2half2(__ushort_as_half(0x1EEE));
    const __half2 a = __half2half2(__ushort_as_half(0xC931));
    __half2 v = __hfma2(h, m, a);
    return *reinterpret_cast<uint32_t*>(&v);
}

// Two hash-codebook weights rounded to fp16: half2(value(a), value(b)).
__device__ __forceinline__ uint32_t hash_pair_rounded(uint32_t sa, uint32_t sb, CodebookConst c)
{
    // Sums inside the registers (operand selects of the add, fp16 pipe) and one permute: the other way round, two permutes and one add,
    // loads the integer pipe that bounds the decode.
    const uint32_t xa = hash_pair(sa, c), xb = hash_pair(sb, c);
    const __half2 ha = *reinterpret_cast<const __half2*>(&xa), hb = *reinterpret_cast<const __half2*>(&xb);
    const __half2 a = __hadd2(__low2half2(ha), __high2half2(ha)), b = __hadd2(__low2half2(hb), __high2half2(hb));
    return prmt(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b), 0x5410);
}

// ---------------------------------------------------------------------------------------------- placement

// Element j (0..7) of lane l sits at row 2*(l&3) + (j&1) + 8*((j>>1)&1), column (l>>2) + 8*(j>>2) of the tile.
__device__ __forceinline__ int tile_row(int lane, int j) { return 2 * (lane & 3) + (j & 1) + 8 * ((j >> 1) & 1); }
__device__ __forceinline__ int tile_col(int lane, int j) { return (lane >> 2) + 8 * (j >> 2); }

// ---------------------------------------------------------------------------------------------- Hadamard

// 128-point transform across a warp: lane l holds elements 4l..4l+3.  Unnormalised.
__device__ __forceinline__ void fwht128(float& v0, float& v1, float& v2, float& v3, int lane)
{
    float a0 = v0 + v1, a1 = v0 - v1, a2 = v2 + v3, a3 = v2 - v3;
    v0 = a0 + a2;
    v1 = a1 + a3;
    v2 = a0 - a2;
    v3 = a1 - a3;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        float p0 = __shfl_xor_sync(0xFFFFFFFFu, v0, m);
        float p1 = __shfl_xor_sync(0xFFFFFFFFu, v1, m);
        float p2 = __shfl_xor_sync(0xFFFFFFFFu, v2, m);
        float p3 = __shfl_xor_sync(0xFFFFFFFFu, v3, m);
        const bool upper = (lane & m) != 0;
        v0 = upper ? p0 - v0 : v0 + p0;
        v1 = upper ? p1 - v1 : v1 + p1;
        v2 = upper ? p2 - v2 : v2 + p2;
        v3 = upper ? p3 - v3 : v3 + p3;
    }
}

// The same transform with a row spread over FOUR lanes (lane l holds elements 32 * (l & 3) .. + 31 of row l >> 2, eight rows
// per warp): five stages stay inside the lane and only two cross lanes, 64 shuffles for eight rows where the layout above
// needs 160 -- the shuffle unit is what bounds the rotation kernels of the many-row paths.  Same stage order (strides 1, 2, ...,
// 64) and the same sums and differences, so the results are the same bits.
// Pairs of elements travel through the packed fp32 instructions of sm_100 (a - b as fma(b, -1, a): one rounding, the same bits), which
// halves the additions: 280 instructions per eight rows instead of 450.
__device__ __forceinline__ unsigned long long f32x2(float a, float b)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f32x2_split(unsigned long long v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ unsigned long long f32x2_add(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f32x2_fma(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// APART: lanes between the four of a row (1: lane l holds elements of row l >> 2, as above; 8: of row l & 7, elements 32 * (l >> 3) ..).
template <int APART = 1>
__device__ __forceinline__ void fwht128_quad(float (&v)[32], int lane)
{
    unsigned long long p[16];
    const unsigned long long minus = f32x2(-1.f, -1.f);
#pragma unroll
    for (int i = 0; i < 16; i++) p[i] = f32x2(v[2 * i] + v[2 * i + 1], v[2 * i] - v[2 * i + 1]);
#pragma unroll
    for (int stride = 1; stride < 16; stride <<= 1) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if ((i & stride) == 0) {
                const unsigned long long lo = p[i], hi = p[i + stride];
                p[i] = f32x2_add(lo, hi);
                p[i + stride] = f32x2_fma(hi, minus, lo);
            }
        }
    }
#pragma unroll
    for (int m = APART; m < 4 * APART; m <<= 1) {
        const float sign = (lane & m) != 0 ? -1.f : 1.f;
        const unsigned long long sign2 = f32x2(sign, sign);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float a, b;
            f32x2_split(p[i], a, b);
            p[i] = f32x2_fma(p[i], sign2, f32x2(__shfl_xor_sync(0xFFFFFFFFu, a, m), __shfl_xor_sync(0xFFFFFFFFu, b, m)));
        }
    }
#pragma unroll
    for (int i = 0; i < 16; i++) f32x2_split(p[i], v[2 * i], v[2 * i + 1]);
}

// The transform of 16 rows on tensor cores, inputs in fp16: rows g and g + 8 of lane 4 g + t, its elements the 16-byte chunks t, t + 4, t + 8, t + 12 of
// a row (a[.][4 j + w]: elements 2 w, 2 w + 1 of chunk 4 j + t) -- what 16-byte loads of 64 consecutive bytes give.  Four of the seven index bits
// (0, 1, and the lane's 3, 4) are the k of m16n8k16 MMAs, whose right operand is the signs of a 16-point transform, or (SIGNED) these
// times a sign vector: products of two fp16 numbers, exact, so the vector costs nothing.  The other three bits are butterflies between a lane's own
// registers: no shuffles, half the additions, and results in the layout that the inputs had: p[2 j + b][h][row] is elements 4 b + 2 h, 4 b + 2 h + 1
// of chunk 4 j + t.  Unnormalised, sums in fp32; 21 million warp instructions where the same transform by
// butterflies over four lanes per row takes 36 (moe_had_in_kernel, 16384 rows of 2048).
struct Had128Rows {
    unsigned long long p[8][2][2];                           // [group][h][row]: packed pairs

    // s: the sign vector's words, laid out as a row; TWO: there are rows g + 8.
    template <bool SIGNED, bool TWO>
    __device__ __forceinline__ void run(const uint32_t (&a0)[16], const uint32_t (&a1)[16], const uint32_t (&s)[16], int lane)
    {
        const int g = lane >> 2, t = lane & 3;
        const uint32_t mask = (__popc(t & (g >> 1)) & 1 ? 0x80008000u : 0u) ^ (g & 1 ? 0x80000000u : 0u);
        const uint32_t one = 0x3C003C00u ^ mask;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int w = 4 * (i >> 1) + 2 * (i & 1);        // group 2 j + b: words 2 b, 2 b + 1 of chunk j
            const uint32_t b0 = SIGNED ? s[w] ^ mask : one, b1 = SIGNED ? s[w + 1] ^ mask : one;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float c[4];
                // volatile: of the whole warp, it must not sink into a branch that only lanes with a result take
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                             : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                             : "r"(a0[w]), "r"(TWO ? a1[w] : 0u), "r"(a0[w + 1]), "r"(TWO ? a1[w + 1] : 0u), "r"(b0), "r"(h ? b1 ^ 0x80008000u : b1), "f"(0.f));
                p[i][h][0] = f32x2(c[0], c[1]);
                p[i][h][1] = f32x2(c[2], c[3]);
            }
        }
        const unsigned long long minus = f32x2(-1.f, -1.f);
#pragma unroll
        for (int stride = 1; stride < 8; stride <<= 1) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (i & stride) continue;
#pragma unroll
                for (int h = 0; h < 2; h++) {
#pragma unroll
                    for (int r = 0; r < (TWO ? 2 : 1); r++) {
                        const unsigned long long lo = p[i][h][r], hi = p[i + stride][h][r];
                        p[i][h][r] = f32x2_add(lo, hi);
                        p[i + stride][h][r] = f32x2_fma(hi, minus, lo);
                    }
                }
            }
        }
    }
    // Element pair w (0..3) of chunk j of a row.
    __device__ __forceinline__ void pair(int row, int j, int w, float& x, float& y) const { f32x2_split(p[2 * j + (w >> 1)][w & 1][row], x, y); }
    // All 32 elements of a row, chunk by chunk.
    __device__ __forceinline__ void row(int r, float (&v)[32]) const
    {
#pragma unroll
        for (int i = 0; i < 16; i++) pair(r, i >> 2, i & 3, v[2 * i], v[2 * i + 1]);
    }
};

constexpr float HAD_SCALE = 0.08838834764831845f;   // 1 / sqrt(128)

// 32 consecutive halves (64 bytes, 16-byte aligned) as floats.
__device__ __forceinline__ void load_half32(const __half* __restrict__ src, float (&v)[32])
{
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint4 raw = reinterpret_cast<const uint4*>(src)[i];
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __half2 h = *reinterpret_cast<const __half2*>(&w[j]);
            v[8 * i + 2 * j] = __low2float(h);
            v[8 * i + 2 * j + 1] = __high2float(h);
        }
    }
}

// A lane's 32 rotated values -> out[at .. at + 31] = fp16(v * (scale * svh[col ..])), or that value converted to bf16: the
// order of the fused epilogues.
__device__ __forceinline__ void had_out_finish(const float (&v)[32], const __half* __restrict__ svh, int col, void* __restrict__ out, long long at,
                                               int out_bf16)
{
    uint32_t packed[16];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint4 sraw = make_uint4(0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u);       // ones
        if (svh) sraw = reinterpret_cast<const uint4*>(svh + col)[i];
        const uint32_t sw[4] = {sraw.x, sraw.y, sraw.z, sraw.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __half2 sh = *reinterpret_cast<const __half2*>(&sw[j]);
            const __half2 h = __floats2half2_rn(v[8 * i + 2 * j] * (HAD_SCALE * __low2float(sh)), v[8 * i + 2 * j + 1] * (HAD_SCALE * __high2float(sh)));
            if (out_bf16) {
                const __nv_bfloat162 bb = __floats2bfloat162_rn(__low2float(h), __high2float(h));
                packed[4 * i + j] = *reinterpret_cast<const uint32_t*>(&bb);
            } else {
                packed[4 * i + j] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
    }
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + at);
#pragma unroll
    for (int i = 0; i < 4; i++) dst[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
}

}  // namespace exl3
