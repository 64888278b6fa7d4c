// Pair-tile kernel of single steps, forward transforms (pair_tile_impl.cuh).
#include "pair_tile_impl.cuh"

namespace sipfft {

const void *pair_tile_fn_fwd() { return reinterpret_cast<const void *>(pair_tile_kernel<true>); }

}  // namespace sipfft
