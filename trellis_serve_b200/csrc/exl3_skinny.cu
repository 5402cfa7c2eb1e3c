// Host side of the decode GEMV / skinny GEMM: work split, shared-memory plan, dispatch on K.
#include <climits>
#include <cstring>

#include "exl3_skinny_kernel.cuh"

namespace exl3 {

static int g_mode_override = -1;
[[maybe_unused]] static int g_tl_next_slot = 0;

#ifdef EXL3_TIMELINE
__device__ unsigned long long g_timeline[TL_SLOTS][TL_CTAS][TL_POINTS];
static unsigned long long* g_tl_base = nullptr;
extern "C" int exl3_debug_timeline(unsigned long long* host_out, int* next_slot)
{
    if (next_slot) *next_slot = g_tl_next_slot;
    return (int)cudaMemcpyFromSymbol(host_out, g_timeline, sizeof(g_timeline));
}
extern "C" void exl3_debug_timeline_reset(void) { g_tl_next_slot = 0; }
#endif

int gemv_default_mode(int codebook)
{
    if (codebook_family(codebook) == FAM_MUL1) return GEMV_PAIRED;
    return g_mode_override >= 0 ? g_mode_override : GEMV_SPLIT;
}

void gemv_set_mode_override(int mode) { g_mode_override = mode; }

WorkspaceLayout workspace_layout(int rows, int k, int n_total, int n_shards)
{
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const int r = rows < SKINNY_MAX_ROWS ? (rows < 1 ? 1 : rows) : SKINNY_MAX_ROWS;
    WorkspaceLayout w;
    w.err_off = 0;
    w.counters_off = WS_HEADER_BYTES;
    w.xf_off = WS_SCRATCH_OFF;
    w.partials_off = up(w.xf_off + (size_t)n_shards * k * operand_pitch(r) * 2 * sizeof(__half));
    w.total = up(w.partials_off + (size_t)(GEMV_MAX_GRID + n_total / 128) * r * 128 * sizeof(float));
    return w;
}

int skinny_init_device()
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    int rc = skinny_set_attributes_for_k<2>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<3>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<4>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<5>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<6>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<7>(d->max_smem_optin);
    if (rc == EXL3_OK) rc = skinny_set_attributes_for_k<8>(d->max_smem_optin);
    return rc;
}

// Work split and shared-memory plan of one launch; `x`: SK_STREAM or one of the modes that keep a slot of activations per unit.  aligned: CTAs
// may get column blocks or equal parts of them instead of even ranges.  slots: of routed experts, or 0.
static int plan_split(const GemvArgs& a, const DeviceInfo* d, int x, bool aligned, int slots, SkinnyLaunch& l, size_t& smem)
{
    memset(&l, 0, sizeof(l));
    l.a = a;
    l.KG = a.k / 128;
    l.NB = a.n_total / 128;
    const int ctas = d->sm_count < GEMV_MAX_GRID ? d->sm_count : GEMV_MAX_GRID;
    l.deal = sk_deal(l.NB, l.KG, ctas, a.rows, x == SK_ROTATE && a.rows > SK_FUSED_ROWS, INT_MAX, aligned, l.most);
    const size_t most = (size_t)l.most;
    // Stages of whole units, as long as three fit; a short range travels as one copy.  A bulk copy costs a few hundred nanoseconds whatever
    // its size (24 KB of weights or more), and a group of decode warps changes stages every ups / 3 units (2 ups / 3 half units): six units where
    // the rows are resident (17408 x 5120, one row, with half units, against stages of 24 KB: K = 3 25.2 -> 24.6 us, K = 4 23.6 -> 22.9, K = 6 27.1 -> 26.1,
    // K = 8 25.4 -> 24.7), no more than 24 KB, or three units, where they travel with the weights and the first stage is waited for (5120 x 5120, 16 rows,
    // with half units: 18.5 us against 19.1 with six units).
    const size_t w = 2048u * (size_t)a.K, f = (size_t)operand_pitch(a.rows) * (a.mode == GEMV_SPLIT ? 512 : 256);
    const SkRaw raw = sk_raw_planes(x, a.x_glu);
    const size_t planes = x == SK_STREAM ? 0 : (size_t)(raw.planes_const + a.rows * raw.planes_row);
    const size_t fixed = SK_BAR_BYTES + (x == SK_STREAM ? 0 : most * f + planes * (most * 256 + 16)) + (size_t)a.rows * 512 + 1024 + slots * sizeof(int2);
    if (fixed >= (size_t)d->max_smem_optin) return EXL3_ERR_UNSUPPORTED_ROWS;
    const size_t budget = (size_t)d->max_smem_optin - fixed, unit = w + (x == SK_STREAM ? f : 0);
    size_t ups = (24 * 1024 + w - 1) / w;
    if (x != SK_STREAM && ups < 6) ups = 6;
    if (ups > most) ups = most;
    // Three units per stage where groups take whole units (see SkWalk).
    const size_t least = a.rows <= SK_FUSED_ROWS || (a.rows > SK_ROTATE_ROWS && a.rows <= 16) ? SK_GROUPS : 2;
    if (ups < least) ups = least;
    if (ups > most) ups = most;
    while (ups > least && budget / (ups * unit) < 3) ups--;
    size_t stages = budget / (ups * unit);
    if (stages > SK_MAX_STAGES) stages = SK_MAX_STAGES;
    const size_t fills = (most + ups - 1) / ups;
    // One or two rows over a range so long that three stages do not fit beside them: two, if they hold 96 KB or more; with less the weights do not
    // keep up and a rotation launch of its own is the faster way.  5120 x 34816 (74 units per CTA), us, two stages of three units / rotation launch /
    // half units in as many stages of two units as fit: K = 5, two rows normalised 51.6 / 49.9 / 52.0; K = 6, one row normalised 52.8 / 50.8 / 50.1,
    // two rows 51.1 / 48.0 / 50.8, normalised 55.4 / 51.6 / 52.5; K = 7, one row 51.9 / 47.7 / 48.2, normalised 53.5 / 51.0 / 51.4, two rows 53.5 / 47.8 /
    // 51.5; two stages do not fit for two normalised rows at K = 7, 51.4 with the launch, 62.6 with half units, and at K = 8 (47.6 / 57.5 for one, 48.2 / 60.1).
    // A step of four such layers, one row: K = 6 484 / 465 / 472, K = 7 490 / 471 / 478.  With 96 KB (K = 8, one row) the launch takes as long
    // alone and more in a stack of four layers: 380 / 387.5 / 379; K = 7, one row there 418 / 414 / 407.  Two stages of four units (K = 7 50.0, 411 in the
    // stack; 17408 x 5120 from gate | up, K = 8, two rows 29.0 against 27.6 with three) are no better.
    if (x != SK_STREAM && a.rows <= SK_FUSED_ROWS && stages < 3 && stages < fills && stages * ups * w < 96 * 1024) return EXL3_ERR_UNSUPPORTED_ROWS;
    if (stages < 2 && stages < fills) return EXL3_ERR_UNSUPPORTED_ROWS;
    // From three rows up the rotation inside saves a launch (3 us) as long as it is one pass of the decode warps and leaves the ring
    // its three stages: 5120 x 5120, 4 rows: 13.3 against 15.9 us; 17408 x 5120, 4 rows: 34.1 against 29.1 us.
    if (x == SK_ROTATE && a.rows > SK_FUSED_ROWS && (most > SK_DECODE_WARPS || (stages < 3 && stages < fills))) return EXL3_ERR_UNSUPPORTED_ROWS;
    if (stages > fills) stages = fills;
    l.stages = (int)stages;
    l.units_per_stage = (int)ups;
    l.x_off = (uint32_t)(SK_BAR_BYTES + stages * ups * w);
    l.r_off = (uint32_t)(l.x_off + (x == SK_STREAM ? stages * ups : most) * f);
    l.r_plane = (uint32_t)(most * 256 + 16);              // 16 bytes apart in the banks: eight rows are read together
    l.p_off = (uint32_t)(l.r_off + planes * l.r_plane);
    l.list_off = (uint32_t)(l.p_off + (size_t)a.rows * 512);
    // Rows behind the last real one are read from whatever follows (their products are dropped): never past the allocation.
    smem = l.list_off + slots * sizeof(int2) + 1024;
    const CodebookConst c = codebook_const(a.codebook);
    l.mul = c.mul;
    l.add = c.add;
    l.slots = slots;
    l.xf_shard_stride = (long long)l.KG * (long long)f;
    return EXL3_OK;
}

static int plan_skinny(const GemvArgs& a, const DeviceInfo* d, int x, SkinnyLaunch& l, size_t& smem, int slots = 0)
{
    const int rc = plan_split(a, d, x, true, slots, l, smem);
    return rc == EXL3_OK || (l.deal.piece == 1 && l.deal.parts == 0) ? rc : plan_split(a, d, x, false, slots, l, smem);      // the busiest CTA's rows may not fit
}

bool skinny_rotates_input(const GemvArgs& a)
{
    const DeviceInfo* d = current_device_info();
    if (!d || !a.x || !a.suh || a.rotated || a.rows < 1 || a.rows > SK_ROTATE_ROWS || a.k < 128 || a.n_total < 128) return false;
    if (a.rows > SK_FUSED_ROWS && (a.norm_weight || a.res_out || a.x_glu)) return false;
    auto odd = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) != 0; };     // the raw input travels by bulk copies
    if (odd(a.x) || odd(a.suh) || odd(a.norm_weight)) return false;
    SkinnyLaunch l;
    size_t smem;
    return plan_skinny(a, d, a.norm_weight ? SK_NORM : SK_ROTATE, l, smem) == EXL3_OK;
}

static int launch_planned(SkinnyLaunch& l, int x, size_t smem, cudaStream_t st)
{
#ifdef EXL3_TIMELINE
    if (!g_tl_base) cudaGetSymbolAddress(reinterpret_cast<void**>(&g_tl_base), g_timeline);
    l.tl = g_tl_base + (size_t)(g_tl_next_slot++ % TL_SLOTS) * TL_CTAS * TL_POINTS;
#endif
    const int pitch = operand_pitch(l.a.rows);
    switch (l.a.K) {
        case 2: return launch_skinny_for_k<2>(l, pitch, x, smem, st);
        case 3: return launch_skinny_for_k<3>(l, pitch, x, smem, st);
        case 4: return launch_skinny_for_k<4>(l, pitch, x, smem, st);
        case 5: return launch_skinny_for_k<5>(l, pitch, x, smem, st);
        case 6: return launch_skinny_for_k<6>(l, pitch, x, smem, st);
        case 7: return launch_skinny_for_k<7>(l, pitch, x, smem, st);
        case 8: return launch_skinny_for_k<8>(l, pitch, x, smem, st);
    }
    return EXL3_ERR_UNSUPPORTED_K;
}

// One of the two products of a routed-expert layer, every slot with a matrix of its own (see SkSlots): rows of k values -> n columns per slot.
static GemvArgs slots_args(int slots, int k, int n, int glu, int K, int codebook)
{
    GemvArgs a;
    memset(&a, 0, sizeof(a));
    a.K = K;
    a.codebook = codebook;
    a.mode = gemv_default_mode(codebook);
    a.rows = 1;
    a.k = k;
    a.n_total = slots * n;
    a.n_shards = 1;
    a.shard_end_blocks[0] = a.n_total / 128;
    a.out_dtype = EXL3_F16;
    a.x_glu = glu;
    return a;
}

bool skinny_serves_slots(int slots, int hidden, int inter, int K, int codebook)
{
    const DeviceInfo* d = current_device_info();
    if (!d || slots < 1 || hidden < 128 || inter < 128 || K < 2 || K > 8) return false;
    for (int down = 0; down < 2; down++) {
        const int k = down ? inter : hidden, n = down ? hidden : 2 * inter;
        const long long blocks = (long long)slots * (n / 128), units = blocks * (k / 128);
        if (blocks * 128 >= (1ll << 31) || blocks > (long long)WS_MAX_COUNTERS || blocks > 2048 || units > (long long)SK_SLOTS_UNITS * d->sm_count) return false;
        SkinnyLaunch l;
        size_t smem;
        if (plan_skinny(slots_args(slots, k, n, down, K, codebook), d, SK_ROTATE, l, smem, slots) != EXL3_OK) return false;
    }
    return true;
}

int launch_skinny_slots(const void* x, int x_bf16, int per_row, const int* ids, const int* map, int experts, int local, int known, int slots, int k, int n,
                        int shards, int glu, const uint32_t* packed, const __half* suh, const __half* svh, int K, int codebook, __half* out,
                        float* partials, int* counters, int* err, cudaStream_t st)
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    GemvArgs a = slots_args(slots, k, n, glu, K, codebook);
    a.packed = packed;
    a.x = x;
    a.x_bf16 = x_bf16;
    a.suh = suh;
    a.svh = svh;
    a.out = out;
    a.partials = partials;
    a.counters = counters;
    a.err = err;
    SkinnyLaunch l;
    size_t smem = 0;
    if (int rc = plan_skinny(a, d, SK_ROTATE, l, smem, slots)) return rc;
    l.s = {ids, map, experts, local, n / 128, n / 128 / shards, per_row, known, (long long)k * n * K / 32};
    return launch_planned(l, SK_ROTATE, smem, st);
}

int launch_skinny(const GemvArgs& a, cudaStream_t st)
{
    const DeviceInfo* d = current_device_info();
    if (!d) return EXL3_ERR_NOT_INITIALISED;
    if (a.rows < 1 || a.rows > SKINNY_MAX_ROWS) return EXL3_ERR_UNSUPPORTED_ROWS;
    const long long units = (long long)(a.k / 128) * (a.n_total / 128);
    if (units == 0) return EXL3_OK;
    if (units >= (1ll << 30)) return EXL3_ERR_BAD_SHAPE;
    SkinnyLaunch l;
    size_t smem = 0;
    const int x = !a.x ? SK_STREAM : a.norm_weight ? SK_NORM : SK_ROTATE;
    if (int rc = plan_skinny(a, d, x, l, smem)) return rc;
    return launch_planned(l, x, smem, st);
}

}  // namespace exl3
