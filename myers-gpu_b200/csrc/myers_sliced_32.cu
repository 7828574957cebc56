// The bit-sliced kernel (myers_sliced.cuh) for 25 to 32 rows per lane.
#include "myers_sliced.cuh"

namespace myers {
MYERS_SLICED_CLASS(Sliced32, 2)
}  // namespace myers
