// bw_tr_f64_1.cu -- transform launches: 64-bit path, 64-bit coefficients in
// double-precision modular arithmetic, prime set 1 of ArD.
#include "bw_transform.cuh"

namespace bw {

template int bw_set_transform_attrs<ArD<1>, false>();
template int bw_enqueue_transform<ArD<1>, false, true>(bw_ctx*, const uint32_t*, const uint32_t*,
                                                       bool, bool, const HostIO*);

}  // namespace bw
