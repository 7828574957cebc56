// The bit-sliced kernel (myers_sliced.cuh) for reads of more than 1,024 bases: groups of several warps.
#include "myers_sliced.cuh"

namespace myers {
MYERS_SLICED_CLASS(SlicedChain, 3)
}  // namespace myers
