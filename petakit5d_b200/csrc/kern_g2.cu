// The y pass kernels of lengths without a compile-time plan, radices up to 31 (gen_engine.cuh).
#include "pass_kernels.cuh"

void pk_fill_kernels_g2(pkpass::KernelTable& t) { pkpass::RegisterYGen<2, 0>::fill(t); }
