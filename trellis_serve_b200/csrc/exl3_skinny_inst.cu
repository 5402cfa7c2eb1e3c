// Instantiates the decode GEMV / skinny GEMM for one bit rate.  Compiled once per K with -DEXL3_SKINNY_K=<2..8>.
#include "exl3_skinny_kernel.cuh"

#ifndef EXL3_SKINNY_K
#error "compile with -DEXL3_SKINNY_K=<2..8>"
#endif

namespace exl3 {

using SkinnyKernel = void (*)(SkinnyLaunch);

// The instance for an operand pitch, a source of activations and an epilogue; null where there is none (more rows than one or two
// with the normalisation or the residual stream inside, more than eight with the rotation inside).
template <int K, int MODE, int FAM>
static SkinnyKernel instance(int pitch, int x, int residual)
{
    if (pitch == 2) {
        if (x == SK_STREAM) return residual ? skinny_kernel<K, MODE, FAM, 2, SK_STREAM, 1> : skinny_kernel<K, MODE, FAM, 2>;
        if (x == SK_ROTATE) return residual ? skinny_kernel<K, MODE, FAM, 2, SK_ROTATE, 1> : skinny_kernel<K, MODE, FAM, 2, SK_ROTATE>;
        return residual ? nullptr : skinny_kernel<K, MODE, FAM, 2, SK_NORM>;
    }
    if (residual) return nullptr;
    if (x == SK_ROTATE) return pitch == 8 ? skinny_kernel<K, MODE, FAM, 8, SK_ROTATE> : nullptr;
    if (x != SK_STREAM) return nullptr;
    return pitch == 8 ? skinny_kernel<K, MODE, FAM, 8> : pitch == 16 ? skinny_kernel<K, MODE, FAM, 16> : pitch == 32 ? skinny_kernel<K, MODE, FAM, 32>
                                                                                                        : skinny_kernel<K, MODE, FAM, 64>;
}

template <int K>
static SkinnyKernel instance_for(int mode, int family, int pitch, int x, int residual)
{
    if (family == FAM_MUL1) return instance<K, GEMV_PAIRED, FAM_MUL1>(pitch, x, residual);
    return mode == GEMV_SPLIT ? instance<K, GEMV_SPLIT, FAM_HASH>(pitch, x, residual) : instance<K, GEMV_PAIRED, FAM_HASH>(pitch, x, residual);
}

template <int K, int SLOTS>
static SkinnyKernel slots_instance(int mode, int family)
{
    if (family == FAM_MUL1) return skinny_kernel<K, GEMV_PAIRED, FAM_MUL1, 2, SK_ROTATE, 0, SLOTS>;
    return mode == GEMV_SPLIT ? skinny_kernel<K, GEMV_SPLIT, FAM_HASH, 2, SK_ROTATE, 0, SLOTS> : skinny_kernel<K, GEMV_PAIRED, FAM_HASH, 2, SK_ROTATE, 0, SLOTS>;
}

template <>
int launch_skinny_for_k<EXL3_SKINNY_K>(const SkinnyLaunch& l, int pitch, int x, size_t smem, cudaStream_t st)
{
    const int family = codebook_family(l.a.codebook);
    const SkinnyKernel kernel = l.s.map   ? slots_instance<EXL3_SKINNY_K, SK_HELD>(l.a.mode, family)
                                : l.s.ids ? slots_instance<EXL3_SKINNY_K, SK_EACH>(l.a.mode, family)
                                          : instance_for<EXL3_SKINNY_K>(l.a.mode, family, pitch, x, l.a.res_out != nullptr);
    if (!kernel) return EXL3_ERR_UNSUPPORTED_ROWS;
    // Programmatic stream serialization: prologue, weight copies and the first half units overlap the tail of the kernel ahead; the
    // kernel waits (griddepcontrol.wait) before touching anything that kernel wrote.
    return launch_chained(kernel, dim3(l.deal.grid), dim3(SK_THREADS), smem, st, l);
}

template <>
int skinny_set_attributes_for_k<EXL3_SKINNY_K>(int max_smem)
{
    auto opt_in = [&](SkinnyKernel kernel) {
        return cuda_status(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    };
    for (int family : {FAM_HASH, FAM_MUL1})
        for (int mode : {GEMV_SPLIT, GEMV_PAIRED}) {
            if (int rc = opt_in(slots_instance<EXL3_SKINNY_K, SK_EACH>(mode, family))) return rc;
            if (int rc = opt_in(slots_instance<EXL3_SKINNY_K, SK_HELD>(mode, family))) return rc;
            for (int pitch : {2, 8, 16, 32, 64})
                for (int x : {SK_STREAM, SK_ROTATE, SK_NORM})
                    for (int residual : {0, 1}) {
                        const SkinnyKernel kernel = instance_for<EXL3_SKINNY_K>(mode, family, pitch, x, residual);
                        if (!kernel) continue;
                        if (int rc = opt_in(kernel)) return rc;
                    }
        }
    return EXL3_OK;
}

}  // namespace exl3
