// The x / z pass kernels of lengths without a compile-time plan (pass_gen.cuh).
#define PK_GEN_KERNEL
#include "pass_gen.cuh"

void pk_fill_gen(pkpass::GenKernel& k) {
    k.fn[0] = pkpass::k_xzg<false>;
    k.fn[1] = pkpass::k_xzg<true>;
    for (auto& f : k.fn)
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
}
