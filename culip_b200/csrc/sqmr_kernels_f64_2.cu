#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(double, 1, 2)
CULIPX_SQMR_PERSISTENT(double, 2, 2)
}  // namespace persistent

}  // namespace culipx
