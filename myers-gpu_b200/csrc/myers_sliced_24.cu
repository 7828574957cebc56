// The bit-sliced kernel (myers_sliced.cuh) for 17 to 24 rows per lane.
#include "myers_sliced.cuh"

namespace myers {
MYERS_SLICED_CLASS(Sliced24, 1)
}  // namespace myers
