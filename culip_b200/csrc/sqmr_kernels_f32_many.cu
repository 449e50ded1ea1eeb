#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_MANY(float, true)
}  // namespace persistent

}  // namespace culipx
