// Instantiates the persistent LPA kernel for 16 sketch slot(s) (separate unit: parallel build).
#include "rak_lpa.cuh"

namespace rak {
template cudaError_t launch_lpa_slots<16>(const LpaArgs &, int, bool, bool, cudaStream_t, int *);
template cudaError_t resolve_lpa_slots<16>(int, bool, bool, bool, bool, int, const void **, int *);
}
