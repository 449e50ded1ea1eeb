#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(float, 1, 4)
CULIPX_SQMR_PERSISTENT(float, 2, 4)
}  // namespace persistent

}  // namespace culipx
