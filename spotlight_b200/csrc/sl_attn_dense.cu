// The tensor-core decode attention (sl_attn_mma.cuh) without an index list, a module of its own. The 32-layer decode step at 32K keys took
// 807 us with these forms (and the row copy of sl_load.cu) in the decode kernels' modules and 801 - 805 with them apart, where
// 801 - 805 had been measured before either: a difference of at most 1 %, whose cause is not known (the same registers).
#include "sl_attn_mma.cuh"

namespace sl {

int launch_attn_dense(const AttnArgs& a, int G, cudaStream_t s) { return launch_by_shape<false, true>(a, G, s); }

}  // namespace sl
