#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(float, 1, 2)
CULIPX_SQMR_PERSISTENT(float, 2, 2)
}  // namespace persistent

}  // namespace culipx
