// The y pass kernels of lengths without a compile-time plan, radices up to 16 (gen_engine.cuh).
#include "pass_kernels.cuh"

void pk_fill_kernels_g1(pkpass::KernelTable& t) { pkpass::RegisterYGen<1, 0>::fill(t); }
