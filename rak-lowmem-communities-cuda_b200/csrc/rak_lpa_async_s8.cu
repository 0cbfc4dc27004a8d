// Instantiates the asynchronous kernel that keeps its pace for 8 sketch slot(s) (separate unit: parallel build).
#include "rak_lpa_async.cuh"

namespace rak {
template const void *async_kernel<8>(bool, bool, bool);
}
