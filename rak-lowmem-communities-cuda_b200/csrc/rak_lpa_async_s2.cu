// Instantiates the asynchronous kernel that keeps its pace for 2 sketch slot(s) (separate unit: parallel build).
#include "rak_lpa_async.cuh"

namespace rak {
template const void *async_kernel<2>(bool, bool, bool);
}
