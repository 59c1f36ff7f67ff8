// batch.cu -- the batched step's kernels, compiled beside abi.cu.
#define SSB_INSTANCE
#include "instances.cuh"

namespace ssb {
SSB_BATCH_INSTANCES
}
