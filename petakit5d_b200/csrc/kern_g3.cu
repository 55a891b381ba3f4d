// The y, x and z pass kernels of lengths with a prime factor above 31 (stage_direct of fft_engine.cuh).
#include "pass_kernels.cuh"

void pk_fill_kernels_g3(pkpass::KernelTable& t) {
    pkpass::RegisterYGen<3, 0>::fill(t);
    auto fn = pkpass::k_xz<0, PK_TILE_POINTS, true>;
    t.xz[pkpass::kSumsXZ] = fn;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, pkpass::kDirectSmem);
}
