// coop.cu -- the cooperative step's kernels, compiled beside abi.cu.
#define SSB_INSTANCE
#include "instances.cuh"

namespace ssb {
SSB_COOP_INSTANCES
}
