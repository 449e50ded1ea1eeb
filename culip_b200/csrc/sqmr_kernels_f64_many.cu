#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_MANY(double, true)
}  // namespace persistent

}  // namespace culipx
