#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_BATCHED(double)
CULIPX_SQMR_MANY(double, false)
}  // namespace persistent

}  // namespace culipx
