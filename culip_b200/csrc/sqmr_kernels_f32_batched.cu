#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_BATCHED(float)
CULIPX_SQMR_MANY(float, false)
}  // namespace persistent

}  // namespace culipx
