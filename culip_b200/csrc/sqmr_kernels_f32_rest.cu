#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_REST(float)
}  // namespace persistent

}  // namespace culipx
