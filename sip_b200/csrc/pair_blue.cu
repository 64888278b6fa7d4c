// Bluestein transforms in one kernel on pair tiles (pair_tile_impl.cuh).
#include "pair_tile_impl.cuh"

namespace sipfft {

const void *pair_blue_fn() { return reinterpret_cast<const void *>(pair_blue_kernel); }

}  // namespace sipfft
