#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(, double, 4)
}  // namespace persistent

}  // namespace culipx
