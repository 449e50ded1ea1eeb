#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(float, 1, 1)
CULIPX_SQMR_PERSISTENT(float, 2, 1)
}  // namespace persistent

}  // namespace culipx
