#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_PERSISTENT(, float, 4)
}  // namespace persistent

}  // namespace culipx
