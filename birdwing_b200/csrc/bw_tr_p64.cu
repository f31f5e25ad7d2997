// bw_tr_p64.cu -- transform launches: 64-bit path, 32- and 64-bit coefficients.
#include "bw_transform.cuh"

namespace bw {

template int bw_set_transform_attrs<Ar64, false>();
template int bw_enqueue_transform<Ar64, false, false>(bw_ctx*, const uint32_t*, const uint32_t*,
                                                      bool, bool, const HostIO*);
template int bw_enqueue_transform<Ar64, false, true>(bw_ctx*, const uint32_t*, const uint32_t*,
                                                     bool, bool, const HostIO*);

}  // namespace bw
