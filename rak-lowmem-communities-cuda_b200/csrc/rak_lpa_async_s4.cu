// Instantiates the asynchronous kernel that keeps its pace for 4 sketch slot(s) (separate unit: parallel build).
#include "rak_lpa_async.cuh"

namespace rak {
template const void *async_kernel<4>(bool, bool, bool);
}
