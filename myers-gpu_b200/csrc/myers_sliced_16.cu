// The bit-sliced kernel (myers_sliced.cuh) for up to 16 rows per lane.
#include "myers_sliced.cuh"

namespace myers {
MYERS_SLICED_CLASS(Sliced16, 0)
}  // namespace myers
