// Pair-tile kernel of uneven batches, forward transforms (pair_tile_impl.cuh).
#include "pair_tile_impl.cuh"

namespace sipfft {

const void *pair_batch_fn_fwd() { return reinterpret_cast<const void *>(pair_batch_kernel<true>); }

}  // namespace sipfft
