// plain.cu -- the FP32 step of plain rows, compiled beside abi.cu.
#define SSB_INSTANCE
#include "instances.cuh"

namespace ssb {
SSB_PLAIN_INSTANCES
}
