#include "sqmr_persistent.cuh"

namespace culipx {

namespace persistent {
CULIPX_SQMR_REST(double)
}  // namespace persistent

}  // namespace culipx
