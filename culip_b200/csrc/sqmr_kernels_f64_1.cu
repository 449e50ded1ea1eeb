#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(double, 1, 1)
CULIPX_SQMR_PERSISTENT(double, 2, 1)
}  // namespace persistent

}  // namespace culipx
