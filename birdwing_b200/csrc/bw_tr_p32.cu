// bw_tr_p32.cu -- transform launches: 32-bit path, 16-bit coefficients.
#include "bw_transform.cuh"

namespace bw {

template int bw_set_transform_attrs<Ar32, true>();
template int bw_enqueue_transform<Ar32, true, false>(bw_ctx*, const uint32_t*, const uint32_t*,
                                                     bool, bool, const HostIO*);

}  // namespace bw
