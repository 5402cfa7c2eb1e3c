// Caller side of the fused groups in a decode step: the element-wise kernels that sit between the EXL3 linears write the
// NEXT linear's rotated input as tensor-core fragments, once, so that the decode GEMV neither needs a rotation launch of
// its own nor rotates inside every CTA:
//
//   rmsnorm_rotate_kernel   residual += x;  normed = rmsnorm(residual) * weight;  fragments = Had128(fp16(normed) * suh[s])
//   silu_mul_rotate_kernel  act = silu(gate) * up;                                fragments = Had128(fp16(act) * suh)
//
// This is the residual / normalisation fusion around the reference's fused launch (cuda/csrc/exl3_marlin.cu:507-527 is the
// group launch; its engine runs residual add, RMSNorm and the activation as separate kernels ahead of had_in,
// cuda/csrc/exl3_marlin.cu:283-290).  The fragments are those of the stand-alone rotation kernel, bit for bit.
#include "exl3_internal.h"
#include "exl3_ptx.cuh"

namespace exl3 {

constexpr int STEP_THREADS = 1024;
constexpr int STEP_MAX_BLOCKS_PER_WARP = 8;            // 128-column blocks one warp keeps in registers: k <= 32768

__device__ __forceinline__ float to_f32(const void* p, long long i, bool bf16)
{
    return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]) : __half2float(reinterpret_cast<const __half*>(p)[i]);
}

// Rounds to the activation type and returns the rounded value.
__device__ __forceinline__ float round_act(float v, bool bf16) { return bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : __half2float(__float2half_rn(v)); }

__device__ __forceinline__ void store_act4(void* p, long long i, const float (&v)[4], bool bf16)
{
    if (bf16) {
        __nv_bfloat16 b[4];
#pragma unroll
        for (int e = 0; e < 4; e++) b[e] = __float2bfloat16_rn(v[e]);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p) + i) = *reinterpret_cast<uint2*>(b);
    } else {
        __half h[4];
#pragma unroll
        for (int e = 0; e < 4; e++) h[e] = __float2half_rn(v[e]);
        *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(p) + i) = *reinterpret_cast<uint2*>(h);
    }
}

// Four consecutive activations (8-byte aligned) as floats.
__device__ __forceinline__ void load_act4(const void* p, long long i, bool bf16, float (&v)[4])
{
    if (bf16) {
        const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p) + i);
        const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), c = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(c); v[3] = __high2float(c);
    } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(p) + i);
        const __half2 a = *reinterpret_cast<const __half2*>(&raw.x), c = *reinterpret_cast<const __half2*>(&raw.y);
        v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(c); v[3] = __high2float(c);
    }
}

// A lane's four signs of a 128-column block.
__device__ __forceinline__ uint2 lane_signs(const __half* suh_blk, int lane) { return *reinterpret_cast<const uint2*>(suh_blk + 4 * lane); }

// One warp, one (shard, row, 128 block): a[e] are activation values already rounded to the activation type.  They are
// converted to fp16 as the rotation kernel does, scaled by suh, rotated and stored as fragments.
// mode 1: split (every value twice), mode 2: paired; layouts of had_in_kernel.
__device__ __forceinline__ void rotate_store(const float (&a)[4], uint2 sw, uint32_t* xf, int mode, int s, int kts, int rows, int row, int kg, int lane)
{
    float v[4];
    const __half2 s01 = *reinterpret_cast<const __half2*>(&sw.x), s23 = *reinterpret_cast<const __half2*>(&sw.y);
    v[0] = __half2float(__float2half_rn(a[0])) * __low2float(s01);
    v[1] = __half2float(__float2half_rn(a[1])) * __high2float(s01);
    v[2] = __half2float(__float2half_rn(a[2])) * __low2float(s23);
    v[3] = __half2float(__float2half_rn(a[3])) * __high2float(s23);
    fwht128(v[0], v[1], v[2], v[3], lane);
    uint32_t hv[4];
#pragma unroll
    for (int e = 0; e < 4; e++) hv[e] = __half_as_ushort(__float2half_rn(v[e] * HAD_SCALE));
    const long long at4 = (long long)s * kts * 4 + kg * 32 + lane;
    const int pitch = operand_pitch(rows);
    if (mode == 1)
        reinterpret_cast<uint4*>(xf)[at4 * pitch + row] = make_uint4(hv[0] * 0x10001u, hv[1] * 0x10001u, hv[2] * 0x10001u, hv[3] * 0x10001u);
    else
        reinterpret_cast<uint2*>(xf)[((at4 >> 1) * pitch + row) * 2 + (at4 & 1)] = make_uint2(hv[0] | (hv[1] << 16), hv[2] | (hv[3] << 16));
}

// grid = rows, block = STEP_THREADS.  x [rows, k]; residual [rows, k] or null (in / out); weight [k]; suh [shards, k];
// normed [rows, k] or null.  J = 128-column blocks a warp keeps in registers (k <= J * 4096).
template <int J>
__global__ void __launch_bounds__(STEP_THREADS) rmsnorm_rotate_kernel(const void* __restrict__ x, void* __restrict__ residual,
                                                                       const void* __restrict__ weight, float eps, int bf16,
                                                                       const __half* __restrict__ suh, int shards, int rows, int k,
                                                                       void* __restrict__ normed, uint32_t* __restrict__ xf, int mode,
                                                                       void* __restrict__ residual_out)
{
    __shared__ float part[STEP_THREADS / 32];
    __shared__ float rstd_s;
    const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kgs = k >> 7;
    const bool b = bf16 != 0;
    // The norm weights are constants: they are fetched while the kernel ahead is still finishing.
    float wv[J][4];
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int kg = warp + j * (STEP_THREADS / 32);
        if (kg < kgs) load_act4(weight, kg * 128 + 4 * lane, b, wv[j]);
    }
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    float h[J][4];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int kg = warp + j * (STEP_THREADS / 32);
        if (kg < kgs) {
            const long long i0 = (long long)row * k + kg * 128 + 4 * lane;
            float z[4], r[4];
            load_act4(x, i0, b, z);
            if (residual) {
                load_act4(residual, i0, b, r);
#pragma unroll
                for (int e = 0; e < 4; e++) z[e] = round_act(z[e] + r[e], b);
                store_act4(residual_out ? residual_out : residual, i0, z, b);      // in place unless a second buffer is given
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                h[j][e] = z[e];
                ss += z[e] * z[e];
            }
        }
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, m);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    if (warp == 0) {
        float t = part[lane];                            // 32 warps: one partial per lane, added in a fixed order
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, m);
        if (lane == 0) rstd_s = rsqrtf(t / (float)k + eps);
    }
    __syncthreads();
    const float rstd = rstd_s;
#pragma unroll
    for (int j = 0; j < J; j++) {
        const int kg = warp + j * (STEP_THREADS / 32);
        if (kg < kgs) {                                   // warp-uniform: all lanes take part in the rotation's shuffles
            const long long i0 = (long long)row * k + kg * 128 + 4 * lane;
            float a[4];
#pragma unroll
            for (int e = 0; e < 4; e++) a[e] = round_act(h[j][e] * rstd * wv[j][e], b);
            if (normed) store_act4(normed, i0, a, b);
            for (int s = 0; s < shards; s++) rotate_store(a, lane_signs(suh + (long long)s * k + kg * 128, lane), xf, mode, s, k >> 4, rows, row, kg, lane);
        }
    }
}

// One warp per (row, 128 block of the intermediate width).  gu [rows, 2 * inter] = gate | up.
__global__ void silu_mul_rotate_kernel(const void* __restrict__ gu, int bf16, const __half* __restrict__ suh, int rows, int inter,
                                       void* __restrict__ act, uint32_t* __restrict__ xf, int mode)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const int lane = threadIdx.x & 31;
    const int kgs = inter >> 7;
    const long long item = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= (long long)rows * kgs) return;
    const int kg = (int)(item % kgs), row = (int)(item / kgs);
    const bool b = bf16 != 0;
    float a[4], gv[4], uv[4];
    load_act4(gu, (long long)row * 2 * inter + kg * 128 + 4 * lane, b, gv);
    load_act4(gu, (long long)row * 2 * inter + inter + kg * 128 + 4 * lane, b, uv);
#pragma unroll
    for (int e = 0; e < 4; e++) a[e] = round_act(gv[e] / (1.0f + __expf(-gv[e])) * uv[e], b);
    if (act) store_act4(act, (long long)row * inter + kg * 128 + 4 * lane, a, b);
    rotate_store(a, lane_signs(suh + kg * 128, lane), xf, mode, 0, inter >> 4, rows, row, kg, lane);
}

// z = x (+ res_in, rounded to the activation type) -> res_out, and the sums of squares of z per (row, 128 columns) -> ssq.
// One warp per (row, block).  The start of a chain of residual blocks whose linears carry the stream in their epilogues.
__global__ void residual_ssq_kernel(const void* __restrict__ x, const void* __restrict__ res_in, int bf16, int rows, int k,
                                    void* __restrict__ res_out, float* __restrict__ ssq)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const int lane = threadIdx.x & 31;
    const int kgs = k >> 7;
    const long long item = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= (long long)rows * kgs) return;
    const bool b = bf16 != 0;
    const long long at = (item / kgs) * k + (item % kgs) * 128 + 4 * lane;
    float z[4], r[4];
    load_act4(x, at, b, z);
    if (res_in) {
        load_act4(res_in, at, b, r);
#pragma unroll
        for (int e = 0; e < 4; e++) z[e] = round_act(z[e] + r[e], b);
    }
    if (res_out) store_act4(res_out, at, z, b);
    float ss = z[0] * z[0] + z[1] * z[1] + z[2] * z[2] + z[3] * z[3];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, m);
    if (lane == 0) ssq[item] = ss;
}

// out = z * rsqrt(mean square + eps) * weight, one warp per (row, 128 columns), the mean square from the sums in ssq [rows, k / 128]: the end
// of a chain of residual blocks.  Latency bounds it (5 elementwise and normalisation launches of a framework in its place took 11 us).
__global__ void normed_kernel(const void* __restrict__ z, const float* __restrict__ ssq, const void* __restrict__ weight, float eps, int bf16, int rows, int k,
                              void* __restrict__ out)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const int lane = threadIdx.x & 31, kgs = k >> 7;
    const long long item = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= (long long)rows * kgs) return;
    const bool b = bf16 != 0;
    const int col = (int)(item % kgs) * 128 + 4 * lane;
    float v[4], w[4], sum = 0.f;
    load_act4(z, (item / kgs) * k + col, b, v);
    load_act4(weight, col, b, w);
    for (int i = lane; i < kgs; i += 32) sum += ssq[(item / kgs) * kgs + i];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, m);
    const float rstd = rsqrtf(sum / (float)k + eps);
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = v[e] * rstd * w[e];
    store_act4(out, (item / kgs) * k + col, v, b);
}

int launch_normed(const void* z, const float* ssq, const void* weight, float eps, int bf16, int rows, int k, void* out, cudaStream_t st)
{
    const long long items = (long long)rows * (k / 128);
    if (items == 0) return EXL3_OK;
    return launch_chained(normed_kernel, dim3((unsigned)((items + 7) / 8)), dim3(256), 0, st, z, ssq, weight, eps, bf16, rows, k, out);
}

int launch_residual_ssq(const void* x, const void* res_in, int bf16, int rows, int k, void* res_out, float* ssq, cudaStream_t st)
{
    const long long items = (long long)rows * (k / 128);
    if (items == 0) return EXL3_OK;
    return launch_chained(residual_ssq_kernel, dim3((unsigned)((items + 7) / 8)), dim3(256), 0, st, x, res_in, bf16, rows, k, res_out, ssq);
}

int launch_rmsnorm_rotate(const void* x, void* residual, const void* weight, float eps, int bf16, const __half* suh, int shards, int rows,
                          int k, void* normed, uint32_t* xf, int mode, cudaStream_t st, void* residual_out)
{
    if (rows == 0 || k == 0) return EXL3_OK;
    if ((k >> 7) > STEP_MAX_BLOCKS_PER_WARP * (STEP_THREADS / 32)) return EXL3_ERR_BAD_SHAPE;
    const int per_warp = ((k >> 7) + STEP_THREADS / 32 - 1) / (STEP_THREADS / 32);
    auto kernel = per_warp <= 2 ? rmsnorm_rotate_kernel<2> : per_warp <= 4 ? rmsnorm_rotate_kernel<4> : rmsnorm_rotate_kernel<STEP_MAX_BLOCKS_PER_WARP>;
    return launch_chained(kernel, dim3(rows), dim3(STEP_THREADS), 0, st, x, residual, weight, eps, bf16, suh, shards, rows, k, normed, xf, mode,
                          residual_out);
}

int launch_silu_mul_rotate(const void* gu, int bf16, const __half* suh, int rows, int inter, void* act, uint32_t* xf, int mode,
                           cudaStream_t st)
{
    const long long items = (long long)rows * (inter / 128);
    if (items == 0) return EXL3_OK;
    return launch_chained(silu_mul_rotate_kernel, dim3((unsigned)((items + 7) / 8)), dim3(256), 0, st, gu, bf16, suh, rows, inter, act, xf,
                          mode);
}

}  // namespace exl3

// ------------------------------------------------------------------------------------------------ attention side of the step
//
// Between q|k|v and o a decode step applies the rotary embedding to q and k, appends k and v to the cache and attends over
// the cache.  None of it is quantized arithmetic; it is written here so that the step does not pay a dozen framework
// launches per layer.  Head dimension 128, grouped queries (q_heads a multiple of kv_heads), one new token per sequence.

namespace exl3 {

constexpr int ATT_D = 128;
constexpr int ATT_MAX_GROUP = 8;          // query heads per KV head
constexpr int ATT_WARPS = 16;
constexpr int ATT_TILE = 8;               // cache positions that a warp takes at a time: columns of an m16n8k16 MMA
constexpr int ATT_STAGE = ATT_WARPS * ATT_TILE;          // cache positions of a stage of the ring
constexpr int ATT_MAX_STAGES = 3, ATT_MAX_CLUSTER = 8;

// One thread per (row, head, pair i < 64): x1' = x1 cos - x2 sin, x2' = x2 cos + x1 sin with x1 = x[i], x2 = x[i + 64]
// (the "rotate half" convention).  Query heads are rotated in place in qkv; key heads are rotated into the cache slot
// `pos`, value heads copied there.  cache layout [rows, kv_heads, t_max, 128].
__global__ void rope_append_kernel(void* __restrict__ qkv, int bf16, int rows, int q_heads, int kv_heads, const float* __restrict__ cos_t,
                                   const float* __restrict__ sin_t, void* __restrict__ k_cache, void* __restrict__ v_cache, int t_max,
                                   const int* __restrict__ pos_ptr)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    const int heads = q_heads + 2 * kv_heads;
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * heads * 64) return;
    const int i = (int)(idx & 63), head = (int)((idx >> 6) % heads), row = (int)((idx >> 6) / heads);
    const int pos = *pos_ptr;
    if (pos < 0 || pos >= t_max) return;                          // a caller's error: no such cache slot
    const long long base = ((long long)row * heads + head) * ATT_D;
    const bool b = bf16 != 0;
    const float x1 = to_f32(qkv, base + i, b), x2 = to_f32(qkv, base + i + 64, b);
    auto put = [&](void* dst, long long at, float v) {
        if (b) reinterpret_cast<__nv_bfloat16*>(dst)[at] = __float2bfloat16_rn(v);
        else reinterpret_cast<__half*>(dst)[at] = __float2half_rn(v);
    };
    if (head < q_heads + kv_heads) {
        const float c = cos_t[(long long)pos * 64 + i], s = sin_t[(long long)pos * 64 + i];
        const float y1 = x1 * c - x2 * s, y2 = x2 * c + x1 * s;
        if (head < q_heads) {
            put(qkv, base + i, y1);
            put(qkv, base + i + 64, y2);
        } else {
            const long long at = (((long long)row * kv_heads + (head - q_heads)) * t_max + pos) * ATT_D;
            put(k_cache, at + i, y1);
            put(k_cache, at + i + 64, y2);
        }
    } else {
        const long long at = (((long long)row * kv_heads + (head - q_heads - kv_heads)) * t_max + pos) * ATT_D;
        put(v_cache, at + i, x1);
        put(v_cache, at + i + 64, x2);
    }
}

#ifdef EXL3_TIMELINE
// Measurement build only: thread 0 of every attention CTA stamps %globaltimer; the slot is derived from the cache address.
__device__ unsigned long long g_att_timeline[64][256][8];
extern "C" int exl3_debug_att_timeline(unsigned long long* host_out) { return (int)cudaMemcpyFromSymbol(host_out, g_att_timeline, sizeof(g_att_timeline)); }
#define ATT_STAMP(i)                                                                                                          \
    do {                                                                                                                      \
        if (threadIdx.x == 0) {                                                                                               \
            unsigned long long t_;                                                                                            \
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                                                            \
            g_att_timeline[(unsigned)(reinterpret_cast<unsigned long long>(k_cache) >> 22) & 63][blockIdx.x + gridDim.x * blockIdx.y][i] = t_; \
        }                                                                                                                     \
    } while (0)
#else
#define ATT_STAMP(i) do { } while (0)
#endif

// Dynamic shared memory of a CTA: the ring, then what the warps exchange.
constexpr uint32_t ATT_ROW = ATT_D * 2, ATT_STAGE_BYTES = 2 * ATT_STAGE * ATT_ROW;      // a stage's keys, then its values
struct AttShared {
    float p[ATT_WARPS][ATT_TILE][ATT_MAX_GROUP + 4];     // a warp's probabilities (rows of 48 bytes: the stores of a warp meet all banks)
    float keep[ATT_WARPS][ATT_MAX_GROUP];                // factor of what earlier tiles added
    float m[ATT_WARPS][ATT_MAX_GROUP], l[ATT_WARPS][ATT_MAX_GROUP];
    float sum[ATT_MAX_GROUP][ATT_D];                     // the CTA's result: weighted sums, maxima and normalisers per head
    float max[ATT_MAX_GROUP], den[ATT_MAX_GROUP];
    uint16_t q[ATT_MAX_GROUP][ATT_D + 8];                // queries; rows 16 bytes apart in the banks
    uint16_t row[2][ATT_D];                              // key and value of position `pos`
    uint64_t full[ATT_MAX_STAGES], empty[ATT_MAX_STAGES];
};

template <bool BF16>
__device__ __forceinline__ void att_mma(float (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1)
{
    const uint32_t zero = 0;                             // rows 8 .. 15 of A
    if constexpr (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, {%7, %8}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(zero), "r"(a2), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %5}, {%7, %8}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(zero), "r"(a2), "r"(b0), "r"(b1));
}

// Two 16-bit activations <-> floats.
template <bool BF16>
__device__ __forceinline__ float2 att_unpack(uint32_t w)
{
    if constexpr (BF16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
    else return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool BF16>
__device__ __forceinline__ uint16_t att_round(float v)
{
    if constexpr (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(v));
    else return __half_as_ushort(__float2half_rn(v));
}

// Decode attention of one new token per row.  grid = (CTAs of a cluster, kv_heads, rows): the CTAs of a cluster share the positions of one
// (row, KV head) and its G query heads, evenly and contiguously in tiles of eight.
//
//   * scores by m16n8k16 MMAs: A = the query heads (rows G .. 15 are zero), B = eight keys.  Both are 16-bit values as stored, so the
//     products are exact and the sums fp32; the order of the 128 columns inside the MMAs is the one in which a lane reads 32 consecutive
//     bytes of a key;
//   * probabilities, normalisers and weighted sums in fp32: a lane owns four of the 128 columns and walks the warp's eight values, the
//     probabilities come from shared memory as broadcasts (once each: a 16-byte broadcast takes four cycles of the return path);
//   * every warp keeps its own running maximum; the warps of a CTA are merged in warp order, the CTAs of a cluster in rank order over
//     distributed shared memory: the same bits every time.  The output of a head -- one rotation block of the o projection's input -- is
//     finished by one warp, which also writes the rotated fragments of the linear that follows (suh != null).
//
// Latency bounds it: 2048 positions of 8 KV heads are 8.4 MB, 1.3 us of memory time that passes before the wait for the kernel ahead.  Of
// the 8 us between the end of q|k|v and the start of o (27B shape, 2048 positions, one row) 0.9 are the wait, 0.6 queries and new row, 3.3
// scores and values (17 positions per warp), 0.9 the merge in the CTA, 0.6 the cluster barrier, 1.2 the merge of the cluster and o's
// rotation, 0.8 o's wait.  With one CTA of four warps per 128 positions, a lane per key and a merge through memory by the last CTA to
// count itself in they were 15.6 (scores 4.4, values 2.3, hand-over 2.4, merge 4.6): 8 layers 960 -> 901 us, at 4096 positions 1049 -> 925,
// at 4096 positions and 8 rows 1662 -> 1206.  Running the code once ahead of the wait, for the instruction cache, gained nothing; all of a
// warp's tiles in one pass (scores of three stages, then one maximum) 0.3 % at one row, and lost 9 % at 8 rows and 4096 positions.
// With cos_t / sin_t the kernel also does what rope_append_kernel does, with the same roundings: the queries are rotated as
// they are loaded (qkv itself is left as it is), and the warp that owns cache position `pos` rotates the new key into the
// cache and copies the new value there before it reads them like any other position.
template <int G, bool BF16>
__global__ void __launch_bounds__(ATT_WARPS * 32, 1) decode_attention_kernel(const void* __restrict__ qkv, int q_heads, int kv_heads, void* k_cache, void* v_cache,
                                                                              int t_max, const int* __restrict__ pos_ptr, float scale,
                                                                              const float* __restrict__ cos_t, const float* __restrict__ sin_t, int* err,
                                                                              int rows, void* __restrict__ y_out, const __half* __restrict__ suh,
                                                                              uint32_t* __restrict__ xf, int mode, int stages)
{
    extern __shared__ __align__(128) unsigned char att_smem[];
    AttShared& sh = *reinterpret_cast<AttShared*>(att_smem + (size_t)stages * ATT_STAGE_BYTES);
    ATT_STAMP(0);
    ptx::grid_launch_dependents();
    const int rank = blockIdx.x, ctas = gridDim.x, kvh = blockIdx.y, row = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q4 = lane & 3, n8 = lane >> 2;
    // A position outside the cache is a caller's error: it is reported, the rows that exist are attended over, nothing is appended.
    const int given = *pos_ptr;
    const bool inside = given >= 0 && given < t_max;
    const int pos = inside ? given : given < 0 ? -1 : t_max, T = pos < t_max ? pos + 1 : t_max;       // T: valid cache positions
    const int heads = q_heads + 2 * kv_heads;
    const int all_tiles = (T + ATT_TILE - 1) / ATT_TILE, share = (all_tiles + ctas - 1) / ctas, tile0 = rank * share;
    const int tiles = all_tiles - tile0 < 0 ? 0 : all_tiles - tile0 < share ? all_tiles - tile0 : share;
    const int fills = (tiles + ATT_WARPS - 1) / ATT_WARPS;
    const long long rowbase = ((long long)row * kv_heads + kvh) * t_max;
    // Cache rows below `pos` were written by earlier steps: like weights they are constants of this launch and are requested
    // before the wait for the kernel ahead, so their trip from memory overlaps that kernel's tail; row `pos` itself comes from
    // the kernel ahead or from this kernel's own append and is put in place after the wait.
    auto fetch = [&](int j, int slot) {
        const int first = (tile0 + j * ATT_WARPS) * ATT_TILE, left = (tiles - j * ATT_WARPS) * ATT_TILE;
        int n = left < ATT_STAGE ? left : ATT_STAGE;
        if (n > pos - first) n = pos - first;
        if (n <= 0) {
            ptx::mbar_arrive(&sh.full[slot]);
            return;
        }
        unsigned char* ks = att_smem + (size_t)slot * ATT_STAGE_BYTES;
        const long long at = (rowbase + first) * ATT_ROW;
        ptx::mbar_arrive_expect_tx(&sh.full[slot], 2u * (uint32_t)n * ATT_ROW);
        ptx::bulk_g2s(ks, reinterpret_cast<const unsigned char*>(k_cache) + at, (uint32_t)n * ATT_ROW, &sh.full[slot]);
        ptx::bulk_g2s(ks + ATT_STAGE * ATT_ROW, reinterpret_cast<const unsigned char*>(v_cache) + at, (uint32_t)n * ATT_ROW, &sh.full[slot]);
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; i++) {
            ptx::mbar_init(&sh.full[i], 1);
            ptx::mbar_init(&sh.empty[i], ATT_WARPS);
        }
        ptx::mbar_fence_init();
        for (int j = 0; j < stages && j < fills; j++) fetch(j, j);
    }
    const bool owner = inside && tiles > 0 && pos / ATT_TILE >= tile0 && pos / ATT_TILE < tile0 + tiles;       // of position `pos`
    const int with = tiles < ATT_WARPS ? tiles : ATT_WARPS;       // warps that have positions
    const int mine = rank + ctas * warp;                          // heads are dealt to the CTAs, one warp each, to be finished
    uint2 signs = make_uint2(0u, 0u);                             // constants: requested before the wait
    if (suh && mine < G) signs = lane_signs(suh + (kvh * G + mine) * ATT_D, lane);
    bool failed = false;
    __syncthreads();
    ptx::grid_dependency_wait();
    ATT_STAMP(1);
    // Queries, and the new row: a thread per pair (i, i + 64) of a head.
    {
        const int i = threadIdx.x & 63;
        const uint16_t* src = reinterpret_cast<const uint16_t*>(qkv) + (long long)row * heads * ATT_D;
        float c = 1.f, sn = 0.f;
        if (cos_t && inside) {
            c = cos_t[(long long)pos * 64 + i];
            sn = sin_t[(long long)pos * 64 + i];
        }
        auto rotate = [&](uint32_t a, uint32_t b, uint16_t* to) {
            if (cos_t) {
                const float x1 = att_unpack<BF16>(a).x, x2 = att_unpack<BF16>(b).x;
                to[i] = att_round<BF16>(x1 * c - x2 * sn);
                to[i + 64] = att_round<BF16>(x2 * c + x1 * sn);
            } else {
                to[i] = (uint16_t)a;
                to[i + 64] = (uint16_t)b;
            }
        };
        const int g = threadIdx.x >> 6;                       // ATT_MAX_GROUP heads of 64 threads
        const uint16_t* at = src + (kvh * G + (g < G ? g : 0)) * ATT_D;
        const uint32_t a = at[i], b = at[i + 64];
        if (g < 2 && owner) {                                 // the new key (rotated with the tables), the new value
            const long long cat = (rowbase + pos) * ATT_D;
            uint16_t* cache = reinterpret_cast<uint16_t*>(g == 0 ? k_cache : v_cache) + cat;
            const uint16_t* kv = cos_t ? src + (q_heads + kvh + g * kv_heads) * ATT_D : cache;
            const uint32_t ka = kv[i], kb = kv[i + 64];
            if (g == 0) rotate(ka, kb, sh.row[0]);
            else {
                sh.row[1][i] = (uint16_t)ka;
                sh.row[1][i + 64] = (uint16_t)kb;
            }
            if (cos_t) {
                cache[i] = sh.row[g][i];
                cache[i + 64] = sh.row[g][i + 64];
            }
        }
        rotate(g < G ? a : 0u, g < G ? b : 0u, sh.q[g]);
    }
    __syncthreads();
    // As A fragments: lane = head n8, columns 64 i + 16 q4 .. + 15 as eight pairs.
    uint32_t qa[2][8];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint4 w = ptx::lds128(ptx::smem_addr(&sh.q[n8][64 * i + 16 * q4 + 8 * j]));
            qa[i][4 * j] = w.x;
            qa[i][4 * j + 1] = w.y;
            qa[i][4 * j + 2] = w.z;
            qa[i][4 * j + 3] = w.w;
        }
    ATT_STAMP(2);
    float m = -INFINITY, l = 0.f;                             // of head n8; l: this lane's positions only
    float acc[G][4] = {};                                         // columns 4 lane .. + 3 of every head
    int slot = 0;
    uint32_t parity = 0;
#pragma unroll 1
    for (int j = 0; j < fills; j++) {
        const int tile = j * ATT_WARPS + warp;
        if (tile < tiles) {
            const int p0 = (tile0 + tile) * ATT_TILE, n = T - p0 < ATT_TILE ? T - p0 : ATT_TILE;      // positions that exist
            unsigned char* ks = att_smem + (size_t)slot * ATT_STAGE_BYTES + warp * (ATT_TILE * ATT_ROW);
            unsigned char* vs = ks + ATT_STAGE * ATT_ROW;
            if (pos - p0 < ATT_TILE) {                            // this warp owns position `pos`
                reinterpret_cast<uint2*>(ks + (pos - p0) * ATT_ROW)[lane] = reinterpret_cast<const uint2*>(sh.row[0])[lane];
                reinterpret_cast<uint2*>(vs + (pos - p0) * ATT_ROW)[lane] = reinterpret_cast<const uint2*>(sh.row[1])[lane];
                __syncwarp();
            }
            if (!failed && !ptx::mbar_wait(&sh.full[slot], parity)) failed = true;
            // Scores.  Rows of keys are 256 bytes apart: lanes of odd rows read the halves of their 32 bytes in the other order, so that
            // the eight lanes of a quarter warp meet different banks.
            float c[2][4] = {};
            const uint32_t krow = ptx::smem_addr(ks) + n8 * ATT_ROW + q4 * 32, odd = n8 & 1;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint4 u = ptx::lds128(krow + i * 128 + odd * 16), v = ptx::lds128(krow + i * 128 + (odd ^ 1) * 16);
                const uint4 lo = odd ? v : u, hi = odd ? u : v;
                att_mma<BF16>(c[i], qa[i][0], qa[i][1], lo.x, lo.y);
                att_mma<BF16>(c[i], qa[i][2], qa[i][3], lo.z, lo.w);
                att_mma<BF16>(c[i], qa[i][4], qa[i][5], hi.x, hi.y);
                att_mma<BF16>(c[i], qa[i][6], qa[i][7], hi.z, hi.w);
            }
            // This lane: head n8, positions 2 q4 and 2 q4 + 1 of the tile.
            const float s0 = 2 * q4 < n ? (c[0][0] + c[1][0]) * scale : -INFINITY, s1 = 2 * q4 + 1 < n ? (c[0][1] + c[1][1]) * scale : -INFINITY;
            float mx = fmaxf(s0, s1);
            mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
            mx = fmaxf(m, mx);
            const float keep = m == -INFINITY ? 0.f : __expf(m - mx);
            const float base = mx == -INFINITY ? 0.f : mx;        // scores that are all -inf so far have no weight, rather than NaN
            const float e0 = 2 * q4 < n ? __expf(s0 - base) : 0.f, e1 = 2 * q4 + 1 < n ? __expf(s1 - base) : 0.f;
            m = mx;
            l = l * keep + (e0 + e1);
            sh.p[warp][2 * q4][n8] = e0;
            sh.p[warp][2 * q4 + 1][n8] = e1;
            if (q4 == 0) sh.keep[warp][n8] = keep;
            __syncwarp();
            if (j > 0) {
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const float k = sh.keep[warp][g];
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[g][e] *= k;
                }
            }
            const uint32_t vrow = ptx::smem_addr(vs) + lane * 8;
#pragma unroll 4
            for (int u = 0; u < n; u++) {
                const uint2 w = ptx::lds64(vrow + u * ATT_ROW);
                const float2 va = att_unpack<BF16>(w.x), vb = att_unpack<BF16>(w.y);
                float e[ATT_MAX_GROUP];
#pragma unroll
                for (int g = 0; g < G; g += 4) {
                    if (G - g == 1) {
                        e[g] = sh.p[warp][u][g];
                    } else {
                        const float4 f = *reinterpret_cast<const float4*>(&sh.p[warp][u][g]);
                        e[g] = f.x;
                        e[g + 1] = f.y;
                        if (G - g > 2) {
                            e[g + 2] = f.z;
                            e[g + 3] = f.w;
                        }
                    }
                }
#pragma unroll
                for (int g = 0; g < G; g++) {
                    acc[g][0] += e[g] * va.x;
                    acc[g][1] += e[g] * va.y;
                    acc[g][2] += e[g] * vb.x;
                    acc[g][3] += e[g] * vb.y;
                }
            }
            __syncwarp();                                     // the next tile overwrites the probabilities
        }
        if (j + stages < fills) {                     // the ring goes around: more positions than it holds
            if (lane == 0) ptx::mbar_arrive(&sh.empty[slot]);
            if (threadIdx.x == 0) {
                if (!failed && !ptx::mbar_wait(&sh.empty[slot], parity)) failed = true;
                fetch(j + stages, slot);
            }
            __syncwarp();
        }
        if (++slot == stages) {
            slot = 0;
            parity ^= 1;
        }
    }
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 2);
    if (q4 == 0) {
        sh.m[warp][n8] = m;
        sh.l[warp][n8] = l;
    }
    ATT_STAMP(3);
    __syncthreads();                                          // every copy has been waited for and read: the ring's first stage is free
    float* red = reinterpret_cast<float*>(att_smem);              // [warp][G][128]
#pragma unroll
    for (int g = 0; g < G; g++)
        *reinterpret_cast<float4*>(red + ((warp * G + g) * ATT_D + 4 * lane)) = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
    __syncthreads();
    // Weight of part `lane` (a warp of the CTA, a CTA of the cluster) from its maximum; returns the common maximum.
    auto weigh = [&](float part_max, float part_den, float& weight, float& den) {
        float mx = part_max;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        weight = part_max == -INFINITY ? 0.f : __expf(part_max - mx);
        den = weight * part_den;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xFFFFFFFFu, den, o);
        return mx;
    };
    if (warp < G) {
        float weight, den;
        const float mx = weigh(lane < with ? sh.m[lane][warp] : -INFINITY, lane < with ? sh.l[lane][warp] : 0.f, weight, den);
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int w = 0; w < with; w++) {
            const float f = __shfl_sync(0xFFFFFFFFu, weight, w);
            const float4 a = *reinterpret_cast<const float4*>(red + ((w * G + warp) * ATT_D + 4 * lane));
            sum[0] += f * a.x;
            sum[1] += f * a.y;
            sum[2] += f * a.z;
            sum[3] += f * a.w;
        }
        *reinterpret_cast<float4*>(&sh.sum[warp][4 * lane]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
        if (lane == 0) {
            sh.max[warp] = mx;
            sh.den[warp] = den;
        }
    }
    ATT_STAMP(4);
    if (ctas > 1) ptx::cluster_sync_all();
    else __syncthreads();
    ATT_STAMP(5);
    if (mine < G) {
        float4 a[ATT_MAX_CLUSTER];
#pragma unroll
        for (int c = 0; c < ATT_MAX_CLUSTER; c++)
            if (c < ctas) a[c] = ptx::ld_shared_cluster_f32x4(&sh.sum[mine][4 * lane], c);
        float weight, den;
        weigh(lane < ctas ? ptx::ld_shared_cluster_f32(&sh.max[mine], lane) : -INFINITY, lane < ctas ? ptx::ld_shared_cluster_f32(&sh.den[mine], lane) : 0.f, weight, den);
        float num[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < ATT_MAX_CLUSTER; c++)
            if (c < ctas) {
                const float f = __shfl_sync(0xFFFFFFFFu, weight, c);
                num[0] += f * a[c].x;
                num[1] += f * a[c].y;
                num[2] += f * a[c].z;
                num[3] += f * a[c].w;
            }
        const int qh = kvh * G + mine;
        float y[4];
#pragma unroll
        for (int e = 0; e < 4; e++) y[e] = round_act(num[e] / den, BF16);
        if (y_out) store_act4(y_out, ((long long)row * q_heads + qh) * ATT_D + 4 * lane, y, BF16);
        if (suh) rotate_store(y, signs, xf, mode, 0, (q_heads * ATT_D) >> 4, rows, row, qh, lane);
    }
    ATT_STAMP(7);
    if (failed && lane == 0) atomicExch(err, ATT_ERR_WAIT);
    if (!inside && threadIdx.x == 0) atomicExch(err, ATT_ERR_POSITION);
    if (ctas > 1) ptx::cluster_sync_all();                        // no CTA leaves while its shared memory is being read
}

// The kernels keep their part of the cache in dynamic shared memory beyond the default limit: opted in once per device.
template <int G>
static int attention_opt_in()
{
    const int most = (int)(ATT_MAX_STAGES * ATT_STAGE_BYTES + sizeof(AttShared));
    const int rc = cuda_status(cudaFuncSetAttribute(decode_attention_kernel<G, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    return rc != EXL3_OK ? rc : cuda_status(cudaFuncSetAttribute(decode_attention_kernel<G, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}

int attention_init_device()
{
    int rc = attention_opt_in<1>();
    if (rc == EXL3_OK) rc = attention_opt_in<2>();
    if (rc == EXL3_OK) rc = attention_opt_in<4>();
    if (rc == EXL3_OK) rc = attention_opt_in<5>();
    if (rc == EXL3_OK) rc = attention_opt_in<8>();
    return rc;
}

int launch_rope_append(void* qkv, int bf16, int rows, int q_heads, int kv_heads, const float* cos_t, const float* sin_t, void* k_cache,
                       void* v_cache, int t_max, const int* pos, cudaStream_t st)
{
    const long long items = (long long)rows * (q_heads + 2 * kv_heads) * 64;
    if (items == 0) return EXL3_OK;
    return launch_chained(rope_append_kernel, dim3((unsigned)((items + 255) / 256)), dim3(256), 0, st, qkv, bf16, rows, q_heads, kv_heads, cos_t,
                          sin_t, k_cache, v_cache, t_max, pos);
}

template <int G>
static int launch_attention_g(const void* qkv, int bf16, int rows, int q_heads, int kv_heads, void* k_cache, void* v_cache, int t_max,
                              const int* pos, float scale, const float* cos_t, const float* sin_t, int* err, void* out, const __half* suh,
                              uint32_t* xf, int mode, cudaStream_t st)
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    // CTAs that share a (row, KV head): as many as a portable cluster holds, while every one has 64 positions and more to look at and all
    // CTAs of the launch fit on the chip together (a CTA with a full ring has an SM for itself).  No more than eight, however long the
    // context: one row of one KV head keeps 8 of the SMs busy and grows by 1.37 us per 1024 positions (5 query heads; 1.68 with 8).  Chained
    // launches, us, against one CTA per 128 positions merged through memory, whose merge grew with the context as well: one KV head, 5
    // query heads, 4096 / 8192 / 32768 / 131072 positions 8.6 / 14.1 / 47.0 / 178 (12.8 / 23.0 / 73.4 / 285), 8 query heads 9.8 / 16.7 /
    // 57.1 / 219 (18.3 / 28.2 / 82.9 / 324), 8 KV heads of 5 9.1 / 14.7 / 48.1 / 181 (16.6 / 37.0 / 144 / 587).
    const int tiles = (t_max + ATT_TILE - 1) / ATT_TILE;
    int ctas = ATT_MAX_CLUSTER;
    while (ctas > 1 && ((long long)rows * kv_heads * ctas > d->sm_count || tiles < 8 * ctas)) ctas /= 2;
    const int share = (tiles + ctas - 1) / ctas;
    int stages = (share + ATT_WARPS - 1) / ATT_WARPS;
    if (stages > ATT_MAX_STAGES) stages = ATT_MAX_STAGES;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, kv_heads, rows);
    cfg.blockDim = dim3(ATT_WARPS * 32);
    cfg.dynamicSmemBytes = stages * (size_t)ATT_STAGE_BYTES + sizeof(AttShared);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    auto* const kernel = bf16 ? decode_attention_kernel<G, true> : decode_attention_kernel<G, false>;
    return cuda_status(cudaLaunchKernelEx(&cfg, kernel, qkv, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, rows, out, suh, xf, mode,
                                          stages));
}

int launch_decode_attention(const void* qkv, int bf16, int rows, int q_heads, int kv_heads, void* k_cache, void* v_cache, int t_max,
                            const int* pos, float scale, const float* cos_t, const float* sin_t, int* err, void* out, const __half* suh,
                            uint32_t* xf, int mode, cudaStream_t st)
{
    if (rows == 0) return EXL3_OK;
    if (kv_heads < 1 || q_heads % kv_heads) return EXL3_ERR_BAD_SHAPE;
    switch (q_heads / kv_heads) {
        case 1: return launch_attention_g<1>(qkv, bf16, rows, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, out, suh, xf, mode, st);
        case 2: return launch_attention_g<2>(qkv, bf16, rows, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, out, suh, xf, mode, st);
        case 4: return launch_attention_g<4>(qkv, bf16, rows, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, out, suh, xf, mode, st);
        case 5: return launch_attention_g<5>(qkv, bf16, rows, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, out, suh, xf, mode, st);
        case 8: return launch_attention_g<8>(qkv, bf16, rows, q_heads, kv_heads, k_cache, v_cache, t_max, pos, scale, cos_t, sin_t, err, out, suh, xf, mode, st);
    }
    return EXL3_ERR_BAD_SHAPE;
}

}  // namespace exl3
