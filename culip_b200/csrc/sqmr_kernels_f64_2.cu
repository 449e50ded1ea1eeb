#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(, double, 2)
}  // namespace persistent

}  // namespace culipx
